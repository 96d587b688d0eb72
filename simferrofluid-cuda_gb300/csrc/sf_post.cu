// sf_post.cu -- the velocity pipeline after the pressure projection (core/Simulation.cpp:236-241): extrapolation
// of the projected velocity into the air (Extrapolation::Solve) and the collider's boundary condition
// (Collider::Enforce), on device-resident face arrays.
//
// Compiled with -fmad=false: each expression rounds as the reference's C++ does, so the results are bit-identical
// to the CPU restatement on the same inputs.
#include <algorithm>
#include <cmath>
#include <utility>

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
__host__ __device__ __forceinline__ FDims fdims(const Dims &d, int a) {
    return FDims{d.nx + (a == 0), d.ny + (a == 1), d.nz + (a == 2)};
}
__device__ __forceinline__ long long fidx(const FDims &f, int i, int j, int k) {
    return (long long)k + (long long)f.fz * ((long long)j + (long long)f.fy * i);
}

// ------------------------------------------------------------------------------------------------ extrapolation
// The validity of a face grid's faces is held as bits: row (i, j) of axis a has bit_words(fz) words, bit k & 31 of word
// k >> 5 for face (i, j, k); bits past the row's end are zero.  At 256^3 the three axes' bits are 7 MB and stay in L2,
// where a byte a face was 50 MB an axis and sweep.
struct BitRows {
    uint32_t *p[3];
};
__host__ __device__ __forceinline__ int bit_words(int fz) { return (fz + 31) >> 5; }

constexpr int kInitX = 2;  // x planes of a thread of k_extrap_init

// Extrapolation validity (core/Simulation.cpp:237-240) of the three lower faces of cell (i, j, k): fraction < 1 and an
// adjacent cell (face - e_a, face) is liquid; a cell outside the grid is not liquid.  A warp is one word of a row.
// Invalid faces take clear_val here already (when there is a sweep at all): every sweep writes every invalid face,
// and those it gives a value are written again below.  One pass over phi, the fractions and the written faces, all
// comparisons on the bits; two x planes a thread keep enough loads in flight: 161 us at 256^3 (0.87 GB, 0.8 of the
// measured bandwidth), 223 us with one plane, 316 us as a pass an axis.
__global__ void __launch_bounds__(256) k_extrap_init(Dims d, const double *__restrict__ phi, Faces frac, Faces u,
                                                     BitRows valid, double clear_val, int clear) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i0 = blockIdx.z * kInitX;
    if (j > d.ny) return;  // whole warps: a warp is one row
    const bool col = j < d.ny && k < d.nz;
    double p[kInitX + 1], py[kInitX], pz[kInitX], fr[3][kInitX];
#pragma unroll
    for (int q = 0; q <= kInitX; q++) {  // every load first: the pass is bound by their latency otherwise
        const int i = i0 + q - 1;
        p[q] = col && i >= 0 && i < d.nx ? phi[cid(d, i, j, k)] : 1.;
    }
#pragma unroll
    for (int q = 0; q < kInitX; q++) {
        const int i = i0 + q;
        const bool in = i < d.nx;
        py[q] = in && k < d.nz && j > 0 ? phi[cid(d, i, j - 1, k)] : 1.;
        pz[q] = in && j < d.ny && k > 0 && k <= d.nz ? phi[cid(d, i, j, k - 1)] : 1.;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const FDims f = fdims(d, a);
            fr[a][q] = i < f.fx && j < f.fy && k < f.fz ? frac.p[a][fidx(f, i, j, k)] : 1.;
        }
    }
#pragma unroll
    for (int q = 0; q < kInitX; q++) {
        const int i = i0 + q;
        const bool liquid = f64_le0(p[q + 1]);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const FDims f = fdims(d, a);
            const bool row = i < f.fx && j < f.fy, face = row && k < f.fz;
            const bool v = f64_lt1(fr[a][q]) && (liquid || f64_le0(a == 0 ? p[q] : (a == 1 ? py[q] : pz[q])));
            if (face && !v && clear) const_cast<double *>(u.p[a])[fidx(f, i, j, k)] = clear_val;
            const uint32_t bits = __ballot_sync(0xffffffffu, v);
            if (row && threadIdx.x == 0 && (int)blockIdx.x < bit_words(f.fz))
                valid.p[a][(long long)(i * f.fy + j) * bit_words(f.fz) + blockIdx.x] = bits;
        }
    }
}

// One sweep of Extrapolation::Solve (core/Extrapolation.cpp:7-28) on the three face grids (blockIdx.z): invalid faces
// with valid 6-neighbours take their mean (order -x,+x,-y,+y,-z,+z) and become valid.  A thread finds the new faces of
// one word by bit operations on the words around it; the block lists its new faces and takes a thread to each, since a
// word often holds one or two (next to a wall) and an interface fills the words of one row.  Valid faces are never
// written in a sweep, so the in-place update reads only values of the previous sweep.  A sweep touches the bits and
// its layer's faces alone: 98 us an axis and sweep as a pass over all faces, 62 us for the three axes with a warp
// taking its words in turn, 26-65 us with the list (256^3; the first sweep has the most faces).
__global__ void __launch_bounds__(256) k_extrap_sweep(Dims d, Faces u, BitRows valid, BitRows valid1) {
    __shared__ uint32_t near[6][256];
    __shared__ uint16_t list[256 * 32];
    __shared__ int sums[8];
    const int a = blockIdx.z, i = blockIdx.y, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const FDims f = fdims(d, a);
    const int nw = bit_words(f.fz), e0 = blockIdx.x * 256, e = e0 + t;  // word of plane i
    if (i >= f.fx || e0 >= f.fy * nw) return;
    uint32_t fresh = 0;
    if (e < f.fy * nw) {
        const int j = e / nw, w = e - j * nw;
        const uint32_t *b = valid.p[a] + (long long)i * f.fy * nw + e;
        const long long sx = (long long)f.fy * nw;
        const uint32_t m = b[0], lo = w > 0 ? b[-1] : 0u, hi = w < nw - 1 ? b[1] : 0u;
        const uint32_t n[6] = {i > 0 ? b[-sx] : 0u,        i < f.fx - 1 ? b[sx] : 0u, j > 0 ? b[-nw] : 0u,
                               j < f.fy - 1 ? b[nw] : 0u, (m << 1) | (lo >> 31),     (m >> 1) | (hi << 31)};
        const int left = f.fz - 32 * w;
        fresh = (n[0] | n[1] | n[2] | n[3] | n[4] | n[5]) & ~m & (left >= 32 ? 0xffffffffu : (1u << left) - 1u);
        valid1.p[a][(long long)i * f.fy * nw + e] = m | fresh;
#pragma unroll
        for (int o = 0; o < 6; o++) near[o][t] = n[o];
    }
    if (!__syncthreads_or(fresh != 0)) return;
    int upto = __popc(fresh);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int s = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += s;
    }
    if (lane == 31) sums[warp] = upto;
    __syncthreads();
    int at = upto - __popc(fresh), total = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        at += q < warp ? sums[q] : 0;
        total += sums[q];
    }
    for (; fresh; fresh &= fresh - 1) list[at++] = (uint16_t)(t * 32 + __ffs(fresh) - 1);
    __syncthreads();
    double *v = const_cast<double *>(u.p[a]);
    for (int q = t; q < total; q += 256) {
        const int word = list[q] >> 5, bit = list[q] & 31, j = (e0 + word) / nw, w = e0 + word - j * nw;
        const long long fi = fidx(f, i, j, w * 32 + bit);
        const long long st[6] = {-(long long)f.fy * f.fz, (long long)f.fy * f.fz, -f.fz, f.fz, -1, 1};
        double nb[6];
#pragma unroll
        for (int o = 0; o < 6; o++) nb[o] = near[o][word] >> bit & 1u ? v[fi + st[o]] : 0.;
        int cnt = 0;
        double sum = 0;
#pragma unroll
        for (int o = 0; o < 6; o++)
            if (near[o][word] >> bit & 1u) {
                sum += nb[o];
                cnt++;
            }
        v[fi] = sum / cnt;
    }
}

// ------------------------------------------------------------------------------------------------ enforcement
// Collider::Enforce (core/Collider.cpp:75-86) changes the faces with fraction == 1 alone, one in 130 in a walled box, and
// on the z walls one of a row's ends, so a pass with a thread a face leaves 31 lanes of a warp idle there (2.3 ms of
// the 2.7 ms at 256^3).  Three passes instead: list the faces (all three fractions read once), evaluate the list from
// the velocity as it was, write the values: 73, 108 (bound by the FP64 pipe and latency) and 6 us.
struct EnforceLists {
    uint32_t *face[3];    // face indices with fraction == 1
    double *value[3];     // their new velocities
    unsigned *count;      // entries of the three lists
};

// 4096 faces a block; the order of the list's blocks is that of their arrival, which no result depends on.
__global__ void __launch_bounds__(256) k_enforce_list(Dims d, Faces frac, EnforceLists l) {
    __shared__ unsigned sums[8], base;
    const int a = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const FDims f = fdims(d, a);
    const long long n = (long long)f.fx * f.fy * f.fz, first = blockIdx.x * 4096LL + threadIdx.x;
    if (blockIdx.x * 4096LL >= n) return;
    unsigned hit = 0;
#pragma unroll
    for (int q = 0; q < 16; q++)
        if (first + q * 256 < n && f64_is_one(frac.p[a][first + q * 256])) hit |= 1u << q;
    if (!__syncthreads_or(hit != 0)) return;
    const unsigned mine = __popc(hit);
    unsigned upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += t;
    }
    if (lane == 31) sums[warp] = upto;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < 8; w++) {
            const unsigned s = sums[w];
            sums[w] = t;
            t += s;
        }
        base = atomicAdd(l.count + a, t);
    }
    __syncthreads();
    unsigned at = base + sums[warp] + upto - mine;
    for (int q = 0; q < 16; q++)
        if (hit >> q & 1u) l.face[a][at++] = (uint32_t)(first + q * 256);
}

// The new velocity of the listed faces: the interpolated old velocity minus its normal component relative to the solid
// velocity (us.p[0] == nullptr: zero).
__global__ void __launch_bounds__(128) k_enforce_eval(Dims d, Origin og, double h, double invh, Faces old, Faces us,
                                                      Faces normal, EnforceLists l) {
    const unsigned n0 = l.count[0], n1 = l.count[1], n2 = l.count[2];
    const long long total = (long long)n0 + n1 + n2;
    for (long long e = blockIdx.x * 128LL + threadIdx.x; e < total; e += gridDim.x * 128LL) {
        const int a = e < n0 ? 0 : (e < (long long)n0 + n1 ? 1 : 2);
        const long long at = e - (a == 0 ? 0 : (a == 1 ? n0 : (long long)n0 + n1));
        const FDims f = fdims(d, a);
        const uint32_t fi = l.face[a][at], row = fi / (uint32_t)f.fz;
        const int c3[3] = {(int)(row / (uint32_t)f.fy), (int)(row % (uint32_t)f.fy), (int)(fi - row * (uint32_t)f.fz)};
        double p[3];
#pragma unroll
        for (int b = 0; b < 3; b++) p[b] = (b == a ? og.o[b] : og.o[b] + h / 2) + (double)c3[b] * h;  // PositionOf
        const GridPoint q = grid_point(og.o, h, invh, p);
        double vel[3], vel0[3], n[3];
#pragma unroll
        for (int b = 0; b < 3; b++) {
            vel[b] = trilinear_face(d, b, q, old.p[b]);
            vel0[b] = us.p[0] ? trilinear_face(d, b, q, us.p[b]) : 0.0;
            n[b] = trilinear_face(d, b, q, normal.p[b]);
        }
        const double nn = f64_sqrt_any((n[0] * n[0] + n[1] * n[1]) + n[2] * n[2]);  // Vector3d::normalized
        if (nn > 0)
#pragma unroll
            for (int b = 0; b < 3; b++) n[b] = f64_div_any(n[b], nn);
        const double dv0 = vel[0] - vel0[0], dv1 = vel[1] - vel0[1], dv2 = vel[2] - vel0[2];
        const double dn = (dv0 * n[0] + dv1 * n[1]) + dv2 * n[2];
        l.value[a][at] = a == 0 ? vel[0] - dn * n[0] : (a == 1 ? vel[1] - dn * n[1] : vel[2] - dn * n[2]);
    }
}

__global__ void __launch_bounds__(256) k_enforce_put(EnforceLists l, Faces u) {
    const int a = blockIdx.y;
    const unsigned n = l.count[a];
    for (unsigned e = blockIdx.x * 256 + threadIdx.x; e < n; e += gridDim.x * 256)
        const_cast<double *>(u.p[a])[l.face[a][e]] = l.value[a][e];
}

// MagneticField::CalculateVertexPressures (core/MagneticField.cpp:37-48) for vertex v: H trilinear at its position,
// p = mu0/2 chi (|H|^2 + chi^2/(4chi+4) (H.n)^2), mu0 = 4e-7 pi (core/MagneticField.cpp:7-8).  The two factors that
// depend on chi alone come from the host (an FP64 division a vertex otherwise): 74 us for 196,608 vertices
// before, 45 us with that and the samples' products on the integer pipe.
__global__ void __launch_bounds__(128) k_vertex_pressures(Dims d, Origin og, double h, double invh, Faces H,
                                                          double scale, double normal_part,
                                                          const double *__restrict__ pos,
                                                          const double *__restrict__ nrm, long long nv,
                                                          double *__restrict__ out) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x) {
        const double p[3] = {pos[3 * v], pos[3 * v + 1], pos[3 * v + 2]};
        const double n[3] = {nrm[3 * v], nrm[3 * v + 1], nrm[3 * v + 2]};
        const GridPoint q = grid_point(og.o, h, invh, p);
        double hv[3];
#pragma unroll
        for (int b = 0; b < 3; b++) hv[b] = trilinear_face(d, b, q, H.p[b]);
        double coeff = (hv[0] * hv[0] + hv[1] * hv[1]) + hv[2] * hv[2];
        const double hn = (hv[0] * n[0] + hv[1] * n[1]) + hv[2] * n[2];
        coeff += normal_part * hn * hn;
        out[v] = scale * coeff;
    }
}

struct EdgeMarks {
    const int32_t *p[3];
};

// The pressure-jump callback of core/Simulation.cpp:216-235 on the faces of the three axes (blockIdx.z): the vertex of edge
// (a, face - e_a) (Contour::VertexIndexOf; edge grid of axis a = cell grid minus e_a, -1 = no vertex) gives
// J = kappa sigma / rho / h dt - p_m / rho / h dt (terms present when their arrays are), 0 without a vertex.
// A warp takes a row, four faces a lane at a time: every mark is loaded before the first jump is stored.  Bound by HBM
// (4 bytes in and 8 out a face): 100 us an axis with one face a thread, 116 us for the three now (256^3).
__global__ void __launch_bounds__(256) k_pressure_jump(Dims d, EdgeMarks em, const double *__restrict__ kappa,
                                                       const double *__restrict__ pm, double sigma, double rho,
                                                       double invh, double dt, Faces jump) {
    const int a = blockIdx.z, i = blockIdx.y, j = blockIdx.x * 8 + threadIdx.y;
    const FDims f = fdims(d, a);
    if (i >= f.fx || j >= f.fy) return;
    const int ex = d.nx - (a == 0), ey = d.ny - (a == 1), ez = d.nz - (a == 2);
    const int ei = i - (a == 0), ej = j - (a == 1);
    const bool row = ei >= 0 && ej >= 0 && ei < ex && ej < ey;
    const int32_t *marks = em.p[a] + ((long long)ei * ey + ej) * ez - (a == 2);  // mark of face k at marks[k]
    double *out = const_cast<double *>(jump.p[a]) + fidx(f, i, j, 0);
    for (int k0 = threadIdx.x; k0 < f.fz; k0 += 128) {
        int idx[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = k0 + 32 * q, ek = k - (a == 2);
            idx[q] = row && ek >= 0 && ek < ez ? marks[k] : -1;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = k0 + 32 * q;
            double pressure = 0;
            if (kappa && idx[q] >= 0) pressure += f64_div_any(kappa[idx[q]] * sigma, rho) * invh * dt;
            if (pm && idx[q] >= 0) pressure -= f64_div_any(pm[idx[q]], rho) * invh * dt;
            if (k < f.fz) out[k] = pressure;
        }
    }
}

// ------------------------------------------------------------------------------------------------ level set
// The first point of a trace is the cell's centre or the face's, whose cells and weights depend on its index along each
// axis alone: a table for the three axes (entry 0 of axis a at OwnTable::first[a]) instead of 36 FP64 operations a
// trace and 45 for the tricubic weights of a cell that does not move.  Positions: 0 on the faces normal to the axis, 1 on
// the cells' centres; grids as in GridPoint.
struct OwnTable {
    int n, first[3];
    int *lo;     // [position][grid][n], then cubic [n]
    double *w;   // [position][grid][lower, upper][n], then cubic [4][n]
    __device__ __forceinline__ AxisPoint point(int pos, int grid, int e) const {
        const int k = pos * 2 + grid;
        AxisPoint p;
        p.lo = lo[k * n + e];
        p.w[0] = w[(2 * k) * n + e];
        p.w[1] = w[(2 * k + 1) * n + e];
        return p;
    }
    __device__ __forceinline__ CubicPoint cubic(int e) const {
        CubicPoint p;
        p.lo = lo[4 * n + e];
#pragma unroll
        for (int q = 0; q < 4; q++) p.w[q] = w[(8 + q) * n + e];
        return p;
    }
};

__global__ void k_own_table(OwnTable t, Origin og, double h, double invh) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x, pos = blockIdx.y;
    if (e >= t.n) return;
    const int a = e >= t.first[2] ? 2 : (e >= t.first[1] ? 1 : 0);
    const double o = a == 0 ? og.o[0] : (a == 1 ? og.o[1] : og.o[2]);
    const double p = (pos == 0 ? o : o + h / 2) + (double)(e - t.first[a]) * h;
#pragma unroll
    for (int grid = 0; grid < 2; grid++) {
        const AxisPoint q = axis_point(p, grid == 0 ? o : o + h / 2, h, invh);
        const int k = pos * 2 + grid;
        t.lo[k * t.n + e] = q.lo;
        t.w[(2 * k) * t.n + e] = q.w[0];
        t.w[(2 * k + 1) * t.n + e] = q.w[1];
    }
    if (pos == 1) {
        const CubicPoint c = cubic_point(p, o + h / 2, h, invh);
        t.lo[4 * t.n + e] = c.lo;
        for (int q = 0; q < 4; q++) t.w[(8 + q) * t.n + e] = c.w[q];
    }
}

// Advection::Trace<2> (core/Advection.h:15-18): TVD Runge-Kutta trace of second order over dt from the face (i, j, k) of
// axis FACE (-1: the cell).  False when the velocity there is exactly zero (the air beyond the extrapolated layers),
// where p + 0 dt is p, the second sample is the first again and the departure point is p.
template <int FACE>
__device__ __forceinline__ bool trace_rk2(const Dims &d, const Faces &u, const OwnTable &own, const Origin &og,
                                          double h, double invh, const int c3[3], double dt, double out[3]) {
    GridPoint g;
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int a = 0; a < 3; a++) g.on[s][a] = own.point(a == FACE ? 0 : 1, s, own.first[a] + c3[a]);
    g.check();
    double v0[3], v1[3], p[3], q[3];
#pragma unroll
    for (int b = 0; b < 3; b++) v0[b] = trilinear_face(d, b, g, u.p[b]);
    if (f64_is_zero(v0[0]) && f64_is_zero(v0[1]) && f64_is_zero(v0[2])) return false;
#pragma unroll
    for (int b = 0; b < 3; b++) {
        p[b] = (b == FACE ? og.o[b] : og.o[b] + h / 2) + (double)c3[b] * h;
        q[b] = p[b] + v0[b] * dt;
    }
    g = grid_point(og.o, h, invh, q);
#pragma unroll
    for (int b = 0; b < 3; b++) v1[b] = trilinear_face(d, b, g, u.p[b]);
#pragma unroll
    for (int b = 0; b < 3; b++) out[b] = p[b] + (v0[b] + v1[b]) * dt / 2;
    return true;
}

// Advection::Solve<2>(levelSet, velocity, dt) (core/Advection.h:40-49): phi at each cell centre's RK2 departure point
// (trace over -dt), by tricubic interpolation of the old phi.
//
// 620 FP64 operations a cell bound it (8.3 ms at 192^3, a quarter of it liquid); with the weights and three in four of
// the products on the integer pipe, the first point from a table and zero velocities cut short, the FP64 pipe (52%
// busy) and the integer pipe (61%) take 2.4 ms, issue the rest.  64 registers: four blocks an SM against three are worth 7%.
__global__ void __launch_bounds__(256, 4) k_advect_levelset(Dims d, Origin og, double h, double invh, Faces u,
                                                            OwnTable own, double dt, const double *__restrict__ phi,
                                                            double *__restrict__ out) {
    __shared__ double xy[16][256];
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const int c3[3] = {i, j, k};
    double q[3];
    CubicPoint c[3];
    if (trace_rk2<-1>(d, u, own, og, h, invh, c3, -dt, q)) {
#pragma unroll
        for (int a = 0; a < 3; a++) c[a] = cubic_point(q[a], og.o[a] + h / 2, h, invh);
    } else {
#pragma unroll
        for (int a = 0; a < 3; a++) c[a] = own.cubic(own.first[a] + c3[a]);
    }
    out[cid(d, i, j, k)] = tricubic(d, phi, c, xy);
}

// Advection::Solve<2>(velocity, velocity, dt) (core/Advection.h:51-59) for the faces of axis A: trilinear
// interpolation of the old face grid A at each face's RK2 departure point.  Bound as k_advect_levelset is: 9.0 ms at
// 160^3 for the three axes with every operation on the FP64 pipe, 1.8 ms now (67% of the FP64 pipe).
template <int A>
__global__ void __launch_bounds__(256, 4) k_advect_velocity(Dims d, Origin og, double h, double invh, Faces u,
                                                            OwnTable own, double dt, double *__restrict__ out) {
    const FDims f = fdims(d, A);
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= f.fz || j >= f.fy) return;
    const int c3[3] = {i, j, k};
    double q[3];
    GridPoint g;
    if (trace_rk2<A>(d, u, own, og, h, invh, c3, -dt, q)) {
#pragma unroll
        for (int b = 0; b < 3; b++)
            g.on[0][b] = g.on[1][b] = axis_point(q[b], b == A ? og.o[b] : og.o[b] + h / 2, h, invh);
    } else {
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int s = b == A ? 0 : 1;
            g.on[0][b] = g.on[1][b] = own.point(s, s, own.first[b] + c3[b]);
        }
    }
    g.check();
    out[fidx(f, i, j, k)] = trilinear_face(d, A, g, u.p[A]);
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
    const double eps = f64_mul<false, false>(f64_sqr<true>(top), 1e-6);
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
    return f64_mul<true, false>(f64_div(f64_mul<false>(alpha1, phix1) + f64_mul<false>(alpha2, phix2) +
                                           f64_mul<false>(alpha3, phix3), sum), invdx);
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
    const unsigned zb = (unsigned)(d.nz + kRz - 1) / kRz, yb = blockIdx.x / zb;  // reinit_grid
    const int k0 = (int)(blockIdx.x - yb * zb) * kRz, j0 = (int)yb * kRy, i0 = blockIdx.y * kRx;
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
    const bool neg = f64_lt0(fc);
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
                    if (f64_lt0(v) == (left == neg)) p0 = f64_sqr(v);
                }
                if (left && right) queue[atomicAdd(&queued, 1)] = (uint16_t)(a * 256 + tid);
            } else {
                double v = weno_plain(dv[0], dv[1], dv[2], dv[3], dv[4], invdx);
                if (f64_lt0(v) == neg) p0 = v * v;
                v = weno_plain(dv[5], dv[4], dv[3], dv[2], dv[1], invdx);
                if (f64_lt0(v) != neg) p1 = v * v;
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
        if (f64_lt0(v) != f64_lt0(fo)) part[2 * a + 1][t] = f64_sqr(v);
    }
    __syncthreads();
    if (!cell) return;
    double sum = part[0][tid];  // minus side first, as the reference adds them; a zero would leave the sum as it is
#pragma unroll
    for (int q = 1; q < 6; q++)
        if (!f64_is_zero(part[q][tid])) sum += part[q][tid];
    sum = f64_sqrt_any(sum);
    const double sp = h * sum;
    const double sgn = f64_div_any(fc, f64_sqrt_any(fc * fc + sp * sp));
    const double step = fc + dt * sgn * (1. - sum);
    if (STAGE == 0) {
        out[c] = step;
    } else if (STAGE == 1) {
        out[c] = (phi[c] * 3 + step) / 4;
    } else {
        out[c] = f64_third_any(phi[c] + step * 2);
    }
}

// z and y tiles share x: 65,535 tiles of four rows in a launch's y would refuse a grid that the other kernels take
inline dim3 reinit_grid(const Dims &d) {
    return dim3((unsigned)((d.nz + kRz - 1) / kRz) * ((d.ny + kRy - 1) / kRy), (d.nx + kRx - 1) / kRx);
}

inline dim3 cell_grid(const Dims &d) { return dim3((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx); }
}  // namespace

namespace {
// The table in `work` (advect_table_bytes), filled on the stream.
OwnTable own_table(cudaStream_t st, const Dims &d, const Origin &og, double h, void *work) {
    OwnTable t;
    t.first[0] = 0;
    t.first[1] = d.nx + 1;
    t.first[2] = d.nx + d.ny + 2;
    t.n = d.nx + d.ny + d.nz + 3;
    t.w = (double *)work;
    t.lo = (int *)(t.w + 12 * (size_t)t.n);
    k_own_table<<<dim3((t.n + 127) / 128, 2), 128, 0, st>>>(t, og, h, 1 / h);
    return t;
}
}  // namespace

size_t advect_table_bytes(const Dims &d) {
    return (12 * sizeof(double) + 5 * sizeof(int)) * ((size_t)d.nx + d.ny + d.nz + 3);
}

void launch_advect_levelset(cudaStream_t st, const Dims &d, const double origin[3], double h, const Faces &u,
                            double dt, const double *phi, double *out, void *work) {
    Origin og{{origin[0], origin[1], origin[2]}};
    const OwnTable own = own_table(st, d, og, h, work);
    k_advect_levelset<<<cell_grid(d), blk2(), 0, st>>>(d, og, h, 1 / h, u, own, dt, phi, out);
}

void launch_advect_velocity(cudaStream_t st, const Dims &d, const double origin[3], double h, const Faces &u,
                            double dt, double *const out[3], void *work) {
    Origin og{{origin[0], origin[1], origin[2]}};
    const OwnTable own = own_table(st, d, og, h, work);
    k_advect_velocity<0><<<face_grid(d, 0), blk2(), 0, st>>>(d, og, h, 1 / h, u, own, dt, out[0]);
    k_advect_velocity<1><<<face_grid(d, 1), blk2(), 0, st>>>(d, og, h, 1 / h, u, own, dt, out[1]);
    k_advect_velocity<2><<<face_grid(d, 2), blk2(), 0, st>>>(d, og, h, 1 / h, u, own, dt, out[2]);
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
    const double mu0 = 4e-7 * 3.141592653589793238462643383279502884;
    const long long blocks = std::min((nv + 127) / 128, 152LL * 32);
    k_vertex_pressures<<<(unsigned)blocks, 128, 0, st>>>(d, og, h, 1 / h, H, mu0 * 0.5 * chi, chi * chi / (4 * chi + 4),
                                                         pos, nrm, nv, out);
}

void launch_pressure_jump(cudaStream_t st, const Dims &d, const int32_t *const edge_mark[3], const double *kappa,
                          const double *pm, double sigma, double rho, double h, double dt, double *const jump[3]) {
    EdgeMarks em{{edge_mark[0], edge_mark[1], edge_mark[2]}};
    const Faces fj{{jump[0], jump[1], jump[2]}};
    k_pressure_jump<<<dim3((d.ny + 8) / 8, d.nx + 1, 3), blk2(), 0, st>>>(d, em, kappa, pm, sigma, rho, 1 / h, dt, fj);
}

size_t extrapolate_bits_bytes(const Dims &d, int a) {
    const FDims f = fdims(d, a);
    return 4 * (size_t)f.fx * f.fy * bit_words(f.fz);
}

void launch_extrapolate(cudaStream_t st, const Dims &d, const double *phi, const Faces &frac, double *const u[3],
                        uint32_t *const bits[3], uint32_t *const bits1[3], double clear_val, int max_steps) {
    const Faces fu{{u[0], u[1], u[2]}};
    BitRows v0{{bits[0], bits[1], bits[2]}}, v1{{bits1[0], bits1[1], bits1[2]}};
    const dim3 nodes((d.nz + 32) / 32, (d.ny + 8) / 8, (d.nx + kInitX) / kInitX);
    k_extrap_init<<<nodes, blk2(), 0, st>>>(d, phi, frac, fu, v0, clear_val, max_steps > 0 ? 1 : 0);
    // words of one x plane, the most of the three axes
    const int words = std::max((d.ny + 1) * bit_words(d.nz), d.ny * bit_words(d.nz + 1));
    for (int it = 0; it < max_steps; it++) {
        k_extrap_sweep<<<dim3((words + 255) / 256, d.nx + 1, 3), 256, 0, st>>>(d, fu, v0, v1);
        std::swap(v0, v1);
    }
}

void launch_enforce(cudaStream_t st, const Dims &d, const double origin[3], double h, const Faces &us,
                    const Faces &normal, const Faces &frac, double *const u[3], uint32_t *const face[3],
                    double *const value[3], unsigned *count) {
    Origin og{{origin[0], origin[1], origin[2]}};
    const Faces fu{{u[0], u[1], u[2]}};
    EnforceLists l{{face[0], face[1], face[2]}, {value[0], value[1], value[2]}, count};
    cudaMemsetAsync(count, 0, 3 * sizeof(unsigned), st);
    const long long most = std::max({(long long)(d.nx + 1) * d.ny * d.nz, (long long)d.nx * (d.ny + 1) * d.nz,
                                     (long long)d.nx * d.ny * (d.nz + 1)});
    k_enforce_list<<<dim3((unsigned)((most + 4095) / 4096), 3), 256, 0, st>>>(d, frac, l);
    k_enforce_eval<<<152 * 4, 128, 0, st>>>(d, og, h, 1 / h, fu, us, normal, l);  // 1 / h: Grid::m_InvSpacing
    k_enforce_put<<<dim3(152, 3), 256, 0, st>>>(l, fu);
}

}  // namespace sf
