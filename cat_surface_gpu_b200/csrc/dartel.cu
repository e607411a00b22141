// 2-D DARTEL on the spherical lat-lon sheet, batched, for sm_100a.
//
// Every kernel works on a batch of B independent grids of the same size
// (fields laid out [B][channels][ny][nx], contiguous).  Arithmetic follows
// the reference's torch path operation by operation
// (src/cat_surface_gpu/dartel_grid.py, surface_warp.py); this file is
// compiled with --fmad=false so each multiply and add rounds once, which
// makes float64 and float32 results bit-identical to a sequential
// restatement with the same association order.
//
// Boundary rule (dartel_grid.py:190-208): x periodic, y reflected with
// period 2 ny (ny == 1 collapses y to row 0).  Maps are one-based; Jacobians
// are stored (j00, j10, j01, j11).
//
// The host half of this file orchestrates dartel_step (dartel_grid.py:
// 1420-1616), the membrane full multigrid (1211-1417) and the whole solve
// (surface_warp.py:239-367) as launch sequences on one stream, so a caller
// can capture a complete solve in one CUDA graph.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/catsurf_b200.h"
#include "common.cuh"
#include "errors.h"
#include "pdl.cuh"

namespace {

constexpr int kThreads = 256;

// (the remainders only for an index outside the grid: each costs ~25 instructions)
__device__ __forceinline__ int wrap_x(int ix, int nx) {
    if (static_cast<unsigned>(ix) < static_cast<unsigned>(nx)) return ix;
    int r = ix % nx;
    return r < 0 ? r + nx : r;
}

__device__ __forceinline__ int reflect_y(int iy, int ny) {
    if (static_cast<unsigned>(iy) < static_cast<unsigned>(ny)) return iy;
    if (ny == 1) return 0;
    const int period = 2 * ny;
    int r = iy % period;
    if (r < 0) r += period;
    return r >= ny ? period - r - 1 : r;
}

// Bilinear stencil of dartel_grid.py:348-366 at (x, y) (zero-based).
template <typename T>
struct Stencil {
    int i22, i12, i21, i11;  // flat offsets inside one channel
    T dx1, dx2, dy1, dy2;
    __device__ __forceinline__ Stencil(T x, T y, int nx, int ny) {
        const T fx = floor(x), fy = floor(y);
        const int ix = static_cast<int>(fx), iy = static_cast<int>(fy);
        dx1 = x - static_cast<T>(ix);
        dy1 = y - static_cast<T>(iy);
        dx2 = T(1) - dx1;
        dy2 = T(1) - dy1;
        const int x0 = wrap_x(ix, nx), x1 = wrap_x(ix + 1, nx);
        const int y0 = reflect_y(iy, ny), y1 = reflect_y(iy + 1, ny);
        i22 = y0 * nx + x0;
        i12 = y0 * nx + x1;
        i21 = y1 * nx + x0;
        i11 = y1 * nx + x1;
    }
    __device__ __forceinline__ T interp(const T* f) const {
        return (f[i22] * dx2 + f[i12] * dx1) * dy2 + (f[i21] * dx2 + f[i11] * dx1) * dy1;
    }
};

// c moved by whole periods to within half a period of c22.  Less than a quarter of a period apart the
// quotient's floor is 0 and c itself the result; only samples across the periodic seam divide.
template <typename T>
__device__ __forceinline__ T unwrap(T c, T c22, T period) {
    const T d = c - c22;
    if (fabs(d) < T(0.25) * period) return c;
    return c - floor(d / period + T(0.5)) * period;
}

// The stencil's samples (22, 12, 21, 11) of both channels, all read before the seam tests' branches,
// behind which the second channel's reads would wait for the first's (solve 256 x 128: 4.68 -> 4.59 ms).
template <typename T>
struct Samples {
    T v[2][4];
    __device__ __forceinline__ Samples(const Stencil<T>& st, const T* __restrict__ f, int P) {
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            v[ch][0] = f[ch * P + st.i22];
            v[ch][1] = f[ch * P + st.i12];
            v[ch][2] = f[ch * P + st.i21];
            v[ch][3] = f[ch * P + st.i11];
        }
    }
};

struct Pt {
    int b, x, y, i;  // batch, column, row, flat index in a channel
};

__device__ __forceinline__ bool point(int nx, int ny, Pt& p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nx * ny) return false;
    p.b = blockIdx.y;
    p.i = i;
    p.x = i % nx;
    p.y = i / nx;
    return true;
}

// Neighbour offsets with the boundary rule.
__device__ __forceinline__ int nb(int x, int y, int dx, int dy, int nx, int ny) {
    return reflect_y(y + dy, ny) * nx + wrap_x(x + dx, nx);
}

// ---------------------------------------------------------------- kernels

// map = id + v * s (dartel_grid.py:655-675 / 1644-1645) and
// jac = jacobian_of_displacement(v, s) (624-652); either output may be null.
template <typename T>
__global__ void k_smalldef(const T* __restrict__ v, T* __restrict__ map, T* __restrict__ jac, int nx, int ny, T s,
                           T hs) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    const int P = nx * ny;
    const T* vx = v + static_cast<size_t>(p.b) * 2 * P;
    const T* vy = vx + P;
    if (map) {
        T* m = map + static_cast<size_t>(p.b) * 2 * P;
        m[p.i] = static_cast<T>(p.x + 1) + vx[p.i] * s;
        m[P + p.i] = static_cast<T>(p.y + 1) + vy[p.i] * s;
    }
    if (jac) {
        const int xm = nb(p.x, p.y, -1, 0, nx, ny), xp = nb(p.x, p.y, 1, 0, nx, ny);
        const int ym = nb(p.x, p.y, 0, -1, nx, ny), yp = nb(p.x, p.y, 0, 1, nx, ny);
        T* j = jac + static_cast<size_t>(p.b) * 4 * P;
        j[p.i] = (vx[xm] * T(-1) + vx[xp]) * hs + T(1);
        j[P + p.i] = (vy[xm] * T(-1) + vy[xp]) * hs;
        j[2 * P + p.i] = (vx[ym] * T(-1) + vx[yp]) * hs;
        j[3 * P + p.i] = (vy[ym] * T(-1) + vy[yp]) * hs + T(1);
    }
}

// (c, jc) = (b o a, J_b(a) . J_a) (dartel_grid.py:407-507) at point p, with the
// stencil of a at p; jac pointers may be null.
template <typename T>
__device__ __forceinline__ void compose_at(const Stencil<T>& st, const T* __restrict__ a, const T* __restrict__ ja,
                                           const T* __restrict__ b, const T* __restrict__ jb, T* __restrict__ c,
                                           T* __restrict__ jc, int nx, int ny, const Pt& p) {
    const int P = nx * ny;
    const size_t o2 = static_cast<size_t>(p.b) * 2 * P, o4 = static_cast<size_t>(p.b) * 4 * P;
    T* C = c + o2;
    const Samples<T> f(st, b + o2, P);
#pragma unroll
    for (int ch = 0; ch < 2; ++ch) {
        const T period = static_cast<T>(ch == 0 ? nx : ny);
        const T c22 = f.v[ch][0] - T(1);
        const T c12 = unwrap(f.v[ch][1] - T(1), c22, period);
        const T c21 = unwrap(f.v[ch][2] - T(1), c22, period);
        const T c11 = unwrap(f.v[ch][3] - T(1), c22, period);
        C[ch * P + p.i] = (c22 * st.dx2 + c12 * st.dx1) * st.dy2 + (c21 * st.dx2 + c11 * st.dx1) * st.dy1 + T(1);
    }
    if (jc) {
        const T* JA = ja + o4;
        const T* JB = jb + o4;
        const T jb00 = st.interp(JB), jb01 = st.interp(JB + P), jb10 = st.interp(JB + 2 * P),
                jb11 = st.interp(JB + 3 * P);
        const T ja0 = JA[p.i], ja1 = JA[P + p.i], ja2 = JA[2 * P + p.i], ja3 = JA[3 * P + p.i];
        T* J = jc + o4;
        J[p.i] = jb00 * ja0 + jb10 * ja1;
        J[P + p.i] = jb01 * ja0 + jb11 * ja1;
        J[2 * P + p.i] = jb00 * ja2 + jb10 * ja3;
        J[3 * P + p.i] = jb01 * ja2 + jb11 * ja3;
    }
}

template <typename T>
__global__ void k_compose(const T* __restrict__ a, const T* __restrict__ ja, const T* __restrict__ b,
                          const T* __restrict__ jb, T* __restrict__ c, T* __restrict__ jc, int nx, int ny) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    const int P = nx * ny;
    const T* A = a + static_cast<size_t>(p.b) * 2 * P;
    const Stencil<T> st(A[p.i] - T(1), A[P + p.i] - T(1), nx, ny);
    compose_at(st, a, ja, b, jb, c, jc, nx, ny, p);
}

// jac_div_smalldef (dartel_grid.py:678-720) at one point.
template <typename T>
__device__ __forceinline__ void jacdiv_at(const T* J, const T* vx, const T* vy, const Pt& p, int nx, int ny, T hs,
                                          T out[4]) {
    const int P = nx * ny;
    const int xm = nb(p.x, p.y, -1, 0, nx, ny), xp = nb(p.x, p.y, 1, 0, nx, ny);
    const int ym = nb(p.x, p.y, 0, -1, nx, ny), yp = nb(p.x, p.y, 0, 1, nx, ny);
    const T d00 = (vx[xm] * T(-1) + vx[xp]) * hs + T(1);
    const T d10 = (vy[xm] * T(-1) + vy[xp]) * hs;
    const T d01 = (vx[ym] * T(-1) + vx[yp]) * hs;
    const T d11 = (vy[ym] * T(-1) + vy[yp]) * hs + T(1);
    const T det = d00 * d11 - d01 * d10;
    const T i00 = d11 / det, i10 = -d10 / det, i01 = -d01 / det, i11 = d00 / det;
    const T o00 = J[p.i], o10 = J[P + p.i], o01 = J[2 * P + p.i], o11 = J[3 * P + p.i];
    out[0] = o00 * i00 + o01 * i10;
    out[1] = o10 * i00 + o11 * i10;
    out[2] = o00 * i01 + o01 * i11;
    out[3] = o10 * i01 + o11 * i11;
}

template <typename T>
__global__ void k_jacdiv(const T* __restrict__ jac, const T* __restrict__ v, T* __restrict__ out, int nx, int ny,
                         T hs) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    const int P = nx * ny;
    const T* vx = v + static_cast<size_t>(p.b) * 2 * P;
    T r[4];
    jacdiv_at(jac + static_cast<size_t>(p.b) * 4 * P, vx, vx + P, p, nx, ny, hs, r);
    T* o = out + static_cast<size_t>(p.b) * 4 * P;
    for (int k = 0; k < 4; ++k) o[k * P + p.i] = r[k];
}

// Block-level deterministic sum; partial[b * gridDim.x + blockIdx.x].
template <typename T>
__device__ __forceinline__ void block_sum(T value, T* partial) {
    __shared__ T buf[kThreads];
    buf[threadIdx.x] = value;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) buf[threadIdx.x] = buf[threadIdx.x] + buf[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x] = buf[0];
}

// initialise_objfun (dartel_grid.py:723-775), optionally preceded by
// jac_div_smalldef (dartel_step's use, 1497-1512 / 1546-1561).  weights may
// be null (all ones).  Writes rhs [2], hess [3] and the objective partials.
template <typename T, bool JACDIV>
__global__ void k_objfun(const T* __restrict__ source, const T* __restrict__ target, const T* __restrict__ map,
                         const T* __restrict__ jac, const T* __restrict__ v, const T* __restrict__ weights,
                         T* __restrict__ rhs, T* __restrict__ hess, T* __restrict__ partial, int nx, int ny, T hs) {
    csg::pdl_begin();
    Pt p;
    const bool ok = point(nx, ny, p);
    T contrib = T(0);
    if (ok) {
        const int P = nx * ny;
        const size_t o1 = static_cast<size_t>(p.b) * P;
        const T* src = source + o1;
        const T* M = map + 2 * o1;
        T J[4];
        if (JACDIV) {
            const T* vx = v + 2 * o1;
            jacdiv_at(jac + 4 * o1, vx, vx + P, p, nx, ny, hs, J);
        } else {
            const T* JJ = jac + 4 * o1;
            for (int k = 0; k < 4; ++k) J[k] = JJ[k * P + p.i];
        }
        const Stencil<T> st(M[p.i] - T(1), M[P + p.i] - T(1), nx, ny);
        const T k22 = src[st.i22], k12 = src[st.i12], k21 = src[st.i21], k11 = src[st.i11];
        const T sampled = (k22 * st.dx2 + k12 * st.dx1) * st.dy2 + (k21 * st.dx2 + k11 * st.dx1) * st.dy1;
        const T diff = sampled - target[o1 + p.i];
        const T ddx = (k11 - k21) * st.dy1 + (k12 - k22) * st.dy2;
        const T ddy = (k11 * st.dx1 + k21 * st.dx2) - (k12 * st.dx1 + k22 * st.dx2);
        const T gx = J[0] * ddx + J[1] * ddy;
        const T gy = J[2] * ddx + J[3] * ddy;
        const T w = weights ? weights[o1 + p.i] : T(1);
        T* H = hess + 3 * o1;
        T* R = rhs + 2 * o1;
        H[p.i] = gx * gx * w;
        H[P + p.i] = gy * gy * w;
        H[2 * P + p.i] = gx * gy * w;
        R[p.i] = gx * diff * w;
        R[P + p.i] = gy * diff * w;
        contrib = diff * diff * w;
    }
    if (partial) block_sum(contrib, partial);
}

// One scaling-and-squaring increment (dartel_grid.py:832-893; the fused
// form of dartel_triton.py:345-477) at point p: b_out = b + inc_b, a_out = a +
// inc_a, inc = inc_b (inc may be null).  Out of place (the gathers read b and
// a at other points).  st is the stencil of map at p.
template <typename T>
__device__ __forceinline__ void squaring_at(const Stencil<T>& st, const T* __restrict__ b, const T* __restrict__ a,
                                            const T* __restrict__ map, const T* __restrict__ jac,
                                            T* __restrict__ b_out, T* __restrict__ a_out, T* __restrict__ inc,
                                            int nx, int ny, const Pt& p) {
    const int P = nx * ny;
    const size_t o1 = static_cast<size_t>(p.b) * P;
    const T* J = jac + 4 * o1;
    const T* Bv = b + 2 * o1;
    const T* Av = a + 3 * o1;
    const T j00 = J[p.i], j10 = J[P + p.i], j01 = J[2 * P + p.i], j11 = J[3 * P + p.i];
    const T det = j00 * j11 - j01 * j10;
    const T sbx = st.interp(Bv), sby = st.interp(Bv + P);
    const T sa00 = st.interp(Av), sa11 = st.interp(Av + P), sa01 = st.interp(Av + 2 * P);
    const T ibx = det * (sbx * j00 + sby * j10);
    const T iby = det * (sbx * j01 + sby * j11);
    const T t1 = sa00 * j00 + sa01 * j10;
    const T t2 = sa01 * j00 + sa11 * j10;
    const T t3 = sa00 * j01 + sa01 * j11;
    const T t4 = sa01 * j01 + sa11 * j11;
    const T ia00 = det * (t1 * j00 + t2 * j10);
    const T ia11 = det * (t3 * j01 + t4 * j11);
    const T ia01 = det * (t1 * j01 + t2 * j11);
    T* BO = b_out + 2 * o1;
    T* AO = a_out + 3 * o1;
    BO[p.i] = Bv[p.i] + ibx;
    BO[P + p.i] = Bv[P + p.i] + iby;
    AO[p.i] = Av[p.i] + ia00;
    AO[P + p.i] = Av[P + p.i] + ia11;
    AO[2 * P + p.i] = Av[2 * P + p.i] + ia01;
    if (inc) {
        T* I = inc + 2 * o1;
        I[p.i] = ibx;
        I[P + p.i] = iby;
    }
}

template <typename T>
__global__ void k_squaring(const T* __restrict__ b, const T* __restrict__ a, const T* __restrict__ map,
                           const T* __restrict__ jac, T* __restrict__ b_out, T* __restrict__ a_out,
                           T* __restrict__ inc, int nx, int ny) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    const int P = nx * ny;
    const T* M = map + static_cast<size_t>(p.b) * 2 * P;
    const Stencil<T> st(M[p.i] - T(1), M[P + p.i] - T(1), nx, ny);
    squaring_at(st, b, a, map, jac, b_out, a_out, inc, nx, ny, p);
}

// One squaring step followed by the composition of the map with itself, in one
// pass: (b, a) advance as in k_squaring and (map_out, jac_out) = (map o map,
// J(map) . J).  Both read the same map at the same stencil and neither reads
// what the other writes, so the pass equals the two launches; the increment
// k_squaring would store in map_out is overwritten by the composed map there.
template <typename T>
__global__ void k_squaring_compose(const T* __restrict__ b, const T* __restrict__ a, const T* __restrict__ map,
                                   const T* __restrict__ jac, T* __restrict__ b_out, T* __restrict__ a_out,
                                   T* __restrict__ map_out, T* __restrict__ jac_out, int nx, int ny) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    const int P = nx * ny;
    const T* M = map + static_cast<size_t>(p.b) * 2 * P;
    const Stencil<T> st(M[p.i] - T(1), M[P + p.i] - T(1), nx, ny);
    squaring_at(st, b, a, map, jac, b_out, a_out, static_cast<T*>(nullptr), nx, ny, p);
    compose_at(st, map, jac, map, jac, map_out, jac_out, nx, ny, p);
}

// regularization_operator weights (dartel_grid.py:937-1015), host-computed
// in float64 exactly as the reference forms them, cast to T on use.
//   rtype 1: w00, w01, w10
//   rtype 0: wx0, wy0, wx1, wy1, wx2, wy2, wxy
//   rtype 2: w00, w01, w02, w10, w11, w20
struct RegWeights {
    double w[8];
};

RegWeights reg_weights(const double* params, int rtype) {
    const double sx = params[0], sy = params[1], mu = params[2], lam = params[3], id = params[4];
    const double sx2 = sx * sx, sy2 = sy * sy;
    RegWeights r{};
    if (rtype == 1) {
        r.w[0] = mu * (2.0 * sx2 + 2.0 * sy2) + id;
        r.w[1] = -mu * sy2;
        r.w[2] = -mu * sx2;
    } else if (rtype == 0) {
        r.w[0] = mu * (2.0 * sy2 + 4.0 * sx2) + 2.0 * lam * sx2 + id;
        r.w[1] = mu * (2.0 * sx2 + 4.0 * sy2) + 2.0 * lam * sy2 + id;
        r.w[2] = -(2.0 * mu + lam) * sx2;
        r.w[3] = -(2.0 * mu + lam) * sy2;
        r.w[4] = -mu * sx2;
        r.w[5] = -mu * sy2;
        r.w[6] = 0.25 * (lam + mu) * sx * sy;
    } else {
        const double sx4 = sx2 * sx2, sy4 = sy2 * sy2;
        r.w[0] = mu * (6.0 * sx4 + 6.0 * sy4 + 8.0 * sx2 * sy2) + id;
        r.w[1] = mu * (-4.0 * sx2 * sy2 - 4.0 * sy4);
        r.w[2] = mu * sy4;
        r.w[3] = mu * (-4.0 * sx4 - 4.0 * sx2 * sy2);
        r.w[4] = mu * (2.0 * sx2 * sy2);
        r.w[5] = mu * sx4;
    }
    return r;
}

// Membrane weights as relax_membrane / the Triton kernels form them
// (dartel_grid.py:1113-1116): w00 = mu (2 sx sx + 2 sy sy) + id.
struct MemWeights {
    double w00, w01, w10;
};

MemWeights mem_weights(const double* params) {
    const double sx = params[0], sy = params[1], mu = params[2], id = params[4];
    return {mu * (2.0 * sx * sx + 2.0 * sy * sy) + id, -mu * sy * sy, -mu * sx * sx};
}

template <typename T>
__device__ __forceinline__ void regularise_at(const T* vx, const T* vy, const Pt& p, int nx, int ny, int rtype,
                                              const RegWeights& rw, T out[2]) {
    auto at = [&](const T* f, int dx, int dy) { return f[nb(p.x, p.y, dx, dy, nx, ny)]; };
    const T* f[2] = {vx, vy};
    if (rtype == 1) {
        const T w00 = T(rw.w[0]), w01 = T(rw.w[1]), w10 = T(rw.w[2]);
        for (int c = 0; c < 2; ++c)
            out[c] = w00 * f[c][p.i] + w01 * (at(f[c], 0, -1) + at(f[c], 0, 1)) + w10 * (at(f[c], -1, 0) + at(f[c], 1, 0));
    } else if (rtype == 0) {
        const T wx0 = T(rw.w[0]), wy0 = T(rw.w[1]), wx1 = T(rw.w[2]), wy1 = T(rw.w[3]), wx2 = T(rw.w[4]),
                wy2 = T(rw.w[5]), wxy = T(rw.w[6]);
        const T cross_x = at(vy, -1, -1) - at(vy, -1, 1) - at(vy, 1, -1) + at(vy, 1, 1);
        const T cross_y = at(vx, -1, -1) - at(vx, -1, 1) - at(vx, 1, -1) + at(vx, 1, 1);
        out[0] = wx0 * vx[p.i] + wy2 * (at(vx, 0, -1) + at(vx, 0, 1)) + wx1 * (at(vx, -1, 0) + at(vx, 1, 0)) +
                 wxy * cross_x;
        out[1] = wy0 * vy[p.i] + wy1 * (at(vy, 0, -1) + at(vy, 0, 1)) + wx2 * (at(vy, -1, 0) + at(vy, 1, 0)) +
                 wxy * cross_y;
    } else {
        const T w00 = T(rw.w[0]), w01 = T(rw.w[1]), w02 = T(rw.w[2]), w10 = T(rw.w[3]), w11 = T(rw.w[4]),
                w20 = T(rw.w[5]);
        for (int c = 0; c < 2; ++c) {
            const T* g = f[c];
            out[c] = w00 * g[p.i] + w01 * (at(g, 0, -1) + at(g, 0, 1)) + w02 * (at(g, 0, -2) + at(g, 0, 2)) +
                     w10 * (at(g, -1, 0) + at(g, 1, 0)) +
                     w11 * (at(g, -1, -1) + at(g, 1, -1) + at(g, -1, 1) + at(g, 1, 1)) +
                     w20 * (at(g, -2, 0) + at(g, 2, 0));
        }
    }
}

template <typename T>
__global__ void k_regularise(const T* __restrict__ v, T* __restrict__ out, int nx, int ny, int rtype, RegWeights rw) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    const int P = nx * ny;
    const T* vx = v + static_cast<size_t>(p.b) * 2 * P;
    T r[2];
    regularise_at(vx, vx + P, p, nx, ny, rtype, rw, r);
    T* o = out + static_cast<size_t>(p.b) * 2 * P;
    o[p.i] = r[0];
    o[P + p.i] = r[1];
}

// dartel_step's combination (dartel_grid.py:1575-1594):
//   code 1: rhs = (rhs_f - rhs_r) * s + reg(v), hess = (hess_f + hess_r) * s
//   code 0: rhs = rhs_f * s + reg(v),           hess = hess_f * s
// plus the partial sums of reg(v) . v and rhs . rhs (metrics).
template <typename T>
__global__ void k_combine(const T* __restrict__ rf, const T* __restrict__ rr, const T* __restrict__ hf,
                          const T* __restrict__ hr, const T* __restrict__ v, T* __restrict__ rhs, T* __restrict__ hess,
                          T* __restrict__ partial_reg, T* __restrict__ partial_norm, int nx, int ny, T s, RegWeights rw) {
    csg::pdl_begin();
    Pt p;
    const bool ok = point(nx, ny, p);
    T reg_dot = T(0), norm = T(0);
    if (ok) {
        const int P = nx * ny;
        const size_t o1 = static_cast<size_t>(p.b) * P;
        const T* vx = v + 2 * o1;
        T reg[2];
        regularise_at(vx, vx + P, p, nx, ny, 1, rw, reg);
        for (int c = 0; c < 2; ++c) {
            const T base = rr ? rf[2 * o1 + c * P + p.i] - rr[2 * o1 + c * P + p.i] : rf[2 * o1 + c * P + p.i];
            const T r = base * s + reg[c];
            rhs[2 * o1 + c * P + p.i] = r;
            norm = norm + r * r;
            reg_dot = reg_dot + reg[c] * vx[c * P + p.i];
        }
        for (int c = 0; c < 3; ++c) {
            const T base = hr ? hf[3 * o1 + c * P + p.i] + hr[3 * o1 + c * P + p.i] : hf[3 * o1 + c * P + p.i];
            hess[3 * o1 + c * P + p.i] = base * s;
        }
    }
    block_sum(reg_dot, partial_reg);
    block_sum(norm, partial_norm);
}

// (H + L_membrane) u (dartel_grid.py:1018-1070); with `b`, the residual b - (H + L) u.
// Flat offsets of a point's four neighbours under the boundary rule.
struct Nbr4 {
    int xm, xp, ym, yp;
};

__device__ __forceinline__ Nbr4 neighbours(int x, int y, int nx, int ny) {
    return {nb(x, y, -1, 0, nx, ny), nb(x, y, 1, 0, nx, ny), nb(x, y, 0, -1, nx, ny), nb(x, y, 0, 1, nx, ny)};
}

template <typename T>
__device__ __forceinline__ void membrane_apply_at(const T* __restrict__ hess, const T* __restrict__ u,
                                                  const T* __restrict__ b, T* __restrict__ out, int nx, int ny,
                                                  const RegWeights& rw, const Pt& p) {
    const int P = nx * ny;
    const size_t o1 = static_cast<size_t>(p.b) * P;
    const T* ux = u + 2 * o1;
    const T* H = hess + 3 * o1;
    T reg[2];
    regularise_at(ux, ux + P, p, nx, ny, 1, rw, reg);
    const T u0 = ux[p.i], u1 = ux[P + p.i];
    const T a0 = reg[0] + H[p.i] * u0 + H[2 * P + p.i] * u1;
    const T a1 = reg[1] + H[2 * P + p.i] * u0 + H[P + p.i] * u1;
    T* o = out + 2 * o1;
    if (b) {
        o[p.i] = b[2 * o1 + p.i] - a0;
        o[P + p.i] = b[2 * o1 + P + p.i] - a1;
    } else {
        o[p.i] = a0;
        o[P + p.i] = a1;
    }
}

template <typename T>
__global__ void k_membrane_apply(const T* __restrict__ hess, const T* __restrict__ u, const T* __restrict__ b,
                                 T* __restrict__ out, int nx, int ny, RegWeights rw) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    membrane_apply_at(hess, u, b, out, nx, ny, rw, p);
}

// One red-black half sweep, in place (dartel_grid.py:1187-1208 /
// dartel_triton.py:242-291): cells with ((x + y) & 1) == colour.  Exact for
// even nx and for nx == 1, where every neighbour read is either of the other
// colour or the cell itself.
// relax_at with the neighbour offsets given (o1: the batch element's point offset).
template <typename T>
__device__ __forceinline__ void relax_core(const T* __restrict__ hess, const T* __restrict__ b, T* __restrict__ u,
                                           int P, size_t o1, int i, const Nbr4& n, T w00, T w01, T w10) {
    T* ux = u + 2 * o1;
    T* uy = ux + P;
    const T rx = b[2 * o1 + i] - w01 * (ux[n.ym] + ux[n.yp]) - w10 * (ux[n.xm] + ux[n.xp]);
    const T ry = b[2 * o1 + P + i] - w01 * (uy[n.ym] + uy[n.yp]) - w10 * (uy[n.xm] + uy[n.xp]);
    const T* H = hess + 3 * o1;
    const T dxx = H[i] + w00;
    const T dyy = H[P + i] + w00;
    const T cr = H[2 * P + i];
    const T det = dxx * dyy * T(1.0000000001) - cr * cr;
    const T nxv = (dyy * rx - cr * ry) / det;
    const T nyv = (-cr * rx + dxx * ry) / det;
    ux[i] = nxv;
    uy[i] = nyv;
}

template <typename T>
__device__ __forceinline__ void relax_at(const T* __restrict__ hess, const T* __restrict__ b, T* __restrict__ u,
                                         int nx, int ny, T w00, T w01, T w10, const Pt& p) {
    const int P = nx * ny;
    relax_core(hess, b, u, P, static_cast<size_t>(p.b) * P, p.i, neighbours(p.x, p.y, nx, ny), w00, w01, w10);
}

template <typename T>
__global__ void k_relax(const T* __restrict__ hess, const T* __restrict__ b, T* __restrict__ u, int nx, int ny,
                        int colour, T w00, T w01, T w10) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    if (((p.x + p.y) & 1) != colour) return;
    relax_at(hess, b, u, nx, ny, w00, w01, w10, p);
}

// Direct 2x2 point solve of the coarsest level (dartel_grid.py:1318-1334).
template <typename T>
__global__ void k_point_solve(const T* __restrict__ hess, const T* __restrict__ b, T* __restrict__ u, int P, T id) {
    csg::pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const size_t o1 = static_cast<size_t>(blockIdx.y) * P;
    const T* H = hess + 3 * o1;
    const T dxx = H[i] + id, dyy = H[P + i] + id, cr = H[2 * P + i];
    const T det = dxx * dyy * T(1.0000000001) - cr * cr;
    const T b0 = b[2 * o1 + i], b1 = b[2 * o1 + P + i];
    u[2 * o1 + i] = (dyy * b0 - cr * b1) / det;
    u[2 * o1 + P + i] = (-cr * b0 + dxx * b1) / det;
}

template <typename T>
__device__ __forceinline__ T wt2(T d) {
    const T a = fabs(d);
    const T inner = T(0.75) - a * a;
    const T od = T(1.5) - a;
    const T outer = T(0.5) * od * od;
    return a < T(0.5) ? inner : (a < T(1.5) ? outer : T(0));
}

// Taps of resize_at along one axis for target index t: the three source offsets
// (rows: reflected and scaled by the source row length; columns: periodic) and the
// quadratic B-spline weights, formed as resize_at forms them.
template <typename T>
struct AxisTaps {
    int o[3];  // minus, centre, plus
    T w[3];
};

template <typename T>
__device__ __forceinline__ AxisTaps<T> row_taps(int y, int sny, int tny, int snx) {
    const T yl = (static_cast<T>(y) + T(0.5)) * static_cast<T>(sny) / static_cast<T>(tny) - T(0.5);
    const int yo = static_cast<int>(floor(yl + T(0.5)));
    const T yof = static_cast<T>(yo);
    AxisTaps<T> a;
    a.w[1] = wt2(yof - yl);
    a.w[0] = wt2(yof - T(1) - yl);
    a.w[2] = wt2(yof + T(1) - yl);
    a.o[0] = reflect_y(yo - 1, sny) * snx;
    a.o[1] = reflect_y(yo, sny) * snx;
    a.o[2] = reflect_y(yo + 1, sny) * snx;
    return a;
}

template <typename T>
__device__ __forceinline__ AxisTaps<T> col_taps(int x, int snx, int tnx) {
    const T xl = (static_cast<T>(x) + T(0.5)) * static_cast<T>(snx) / static_cast<T>(tnx) - T(0.5);
    const int xo = static_cast<int>(floor(xl + T(0.5)));
    const T xof = static_cast<T>(xo);
    AxisTaps<T> a;
    a.w[1] = wt2(xof - xl);
    a.w[0] = wt2(xof - T(1) - xl);
    a.w[2] = wt2(xof + T(1) - xl);
    a.o[0] = wrap_x(xo - 1, snx);
    a.o[1] = wrap_x(xo, snx);
    a.o[2] = wrap_x(xo + 1, snx);
    return a;
}

// One target value of the separable resize from its row and column taps (f: the source plane).
template <typename T>
__device__ __forceinline__ T resize_value(const T* __restrict__ f, const AxisTaps<T>& r, const AxisTaps<T>& c) {
    const T im = r.w[0] * f[r.o[0] + c.o[0]] + r.w[1] * f[r.o[1] + c.o[0]] + r.w[2] * f[r.o[2] + c.o[0]];
    const T ic = r.w[0] * f[r.o[0] + c.o[1]] + r.w[1] * f[r.o[1] + c.o[1]] + r.w[2] * f[r.o[2] + c.o[1]];
    const T ip = r.w[0] * f[r.o[0] + c.o[2]] + r.w[1] * f[r.o[1] + c.o[2]] + r.w[2] * f[r.o[2] + c.o[2]];
    return c.w[0] * im + c.w[1] * ic + c.w[2] * ip;
}

// Separable quadratic B-spline resize (dartel_grid.py:239-305), y pass then
// x pass, per target point; `accumulate` adds into dst (prolongation,
// dartel_grid.py:1380-1387).  Fields are [B * C][sny][snx] -> [B * C][tny][tnx].
template <typename T>
__device__ __forceinline__ void resize_at(const T* __restrict__ src, T* __restrict__ dst, int snx, int sny, int tnx,
                                          int tny, int accumulate, int plane, int i) {
    const int x = i % tnx, y = i / tnx;
    const T* f = src + static_cast<size_t>(plane) * snx * sny;
    const T r = resize_value(f, row_taps<T>(y, sny, tny, snx), col_taps<T>(x, snx, tnx));
    T* o = dst + static_cast<size_t>(plane) * tnx * tny;
    o[i] = accumulate ? o[i] + r : r;
}

template <typename T>
__global__ void k_resize(const T* __restrict__ src, T* __restrict__ dst, int snx, int sny, int tnx, int tny,
                         int accumulate) {
    csg::pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tnx * tny) return;
    resize_at(src, dst, snx, sny, tnx, tny, accumulate, static_cast<int>(blockIdx.y), i);
}

// ------------------------------------------------ resident V-cycles (one cluster per grid)
//
// From the finest level whose grid fits the shared memory and registers of one
// thread-block cluster (256 x 128 in float64) on, a whole V-cycle -- all cycles of
// a solve when that is level 0 -- is one launch with one cluster per batch element.
// What bounds a V-cycle here is its chain of ~100 half-sweeps and ~40 residuals and
// transfers, each a few hundred cycles of dependent arithmetic: as separate
// launches, or as tiles that recompute their halos, each link cost 2-4 us.  Inside a
// cluster the neighbours' edge rows are written straight into each other's shared memory and
// a link costs 250-550 ns.  Per V-cycle, against legs of 2-D tiles over one CTA for the
// coarse levels: two 256 x 128 grids 129 -> 56 us in float64 and 123 -> 57 in float32, 64 x 32
// 71 -> 27 us, 32 x 16 47 -> 17 us.  Batches of several waves of clusters take legs on the finer levels
// (see ResidentCosts).  Of the 56 us the first level takes 20, the other split levels 20, the levels of
// CTA 0 17.
//
// Levels above kCoarsePoints points are split by rows over the cluster's CTAs, each
// holding its rows of u with a halo row above and below.  The first such level's system
// and right-hand side are read from global memory at each visit, the others' are in
// shared memory; during a visit they are in registers.  The levels below run on CTA 0
// alone, in teams of 256 and 64 threads and one warp as they shrink.  256 threads of up to
// 255 registers, not 512 of 128: the eight points of a thread (float64: 112 registers) must
// not spill, since shared memory leaves the L1 too small for it (70 us per V-cycle with spills).
// Every point sees the operations of relax_core, membrane_apply_at and
// resize_value in their order, so results equal the separate kernels' bit for bit.

constexpr int kCoarsePoints = 512;  // levels of at most this many points run on one CTA, a unit of two points per thread
constexpr int kMaxLevels = 16;
constexpr int kResidentThreads = 256;
constexpr int kResidentSlots = 4;   // units a thread holds of a split level at most
constexpr int kResidentPoints = 2 * kResidentSlots * kResidentThreads;  // of a CTA's rows of it
constexpr int kMaxCluster = 16;     // 16 CTAs is the largest cluster of the architecture (8 is the portable bound)
// A launch of more CTAs than the device's 148 SMs hold as clusters of 16 uses as few CTAs per grid
// as hold it (64 float64 grids of 128 x 64 per V-cycle: 354 us with 16 CTAs each, 95 with 4; two
// of them: 36 and 55), and in float32 the kernel of 128 registers, two CTAs to an SM (32 grids of
// 256 x 128, resident throughout: 286 -> 243 us; two: 57 and 71).
constexpr int kPairedCtas = 128;

// Both components of a field at a point, moved together.
template <typename T>
struct alignas(2 * sizeof(T)) Pair {
    T x, y;
};

// A point's 2 x 2 system: the Hessian, the determinant relax_core divides by, and its
// correctly rounded reciprocal (0: divide).
template <typename T>
struct PointSystem {
    T h0, h1, h2, det, inv;
};

template <typename T>
__device__ __forceinline__ PointSystem<T> point_system(T h0, T h1, T h2, T w00) {
    PointSystem<T> s{h0, h1, h2, T(0), T(0)};
    const T dxx = h0 + w00, dyy = h1 + w00;
    s.det = dxx * dyy * T(1.0000000001) - h2 * h2;
    if constexpr (sizeof(T) == 8) {
        const unsigned e = (static_cast<unsigned>(__double2hiint(s.det)) >> 20) & 0x7ffu;
        if (e - 623u <= 800u) s.inv = __drcp_rn(s.det);  // 2^-400 <= |det| <= 2^400
    }
    return s;
}

// (a.x / s.det, a.y / s.det).  float64: with y = RN(1 / d) and q within an ulp of a / d,
// RN(q + RN(a - d q) y) is the correctly rounded quotient (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1),
// 1990); q0 = RN(a y) is refined once to come within an ulp.  The exponent bounds
// (2^-500 <= |a| < 2^500 here, s.inv = 0 for an extreme determinant) keep every remainder
// and quotient normal; outside them, and for a = 0, the division itself runs.  Both
// quotients share one test, off their dependency chain: a half-sweep of one warp takes 243
// cycles without a test, 365 with one per quotient, as with the divisions.
template <typename T>
__device__ __forceinline__ Pair<T> quotients(T a0, T a1, const PointSystem<T>& s) {
    if constexpr (sizeof(T) == 8) {
        // biased exponents 523 .. 1522, the sign shifted out
        const unsigned e0 = 2u * static_cast<unsigned>(__double2hiint(a0)) - (523u << 21);
        const unsigned e1 = 2u * static_cast<unsigned>(__double2hiint(a1)) - (523u << 21);
        const double p0 = __dmul_rn(a0, s.inv), p1 = __dmul_rn(a1, s.inv);
        const double q0 = __fma_rn(__fma_rn(-s.det, p0, a0), s.inv, p0);
        const double q1 = __fma_rn(__fma_rn(-s.det, p1, a1), s.inv, p1);
        Pair<T> r{__fma_rn(__fma_rn(-s.det, q0, a0), s.inv, q0), __fma_rn(__fma_rn(-s.det, q1, a1), s.inv, q1)};
        if (e0 >= (1000u << 21) || e1 >= (1000u << 21) || __double2hiint(s.inv) == 0) r = {a0 / s.det, a1 / s.det};
        return r;
    } else {
        return {a0 / s.det, a1 / s.det};
    }
}

template <typename T>
struct Weights {
    T w00, w01, w10;
};

template <typename T>
struct ResidentLevel {
    const T* A;  // Hessian [batch][3][ny][nx]
    T* B;        // right-hand side [batch][2][ny][nx] (the first level's is read)
    T* U;        // solution [batch][2][ny][nx] (the first level's is read and written)
    int nx, ny, lg;   // lg: log2(nx), a power of two on every level
    int rows;         // rows of a CTA's slab at most (0: a level of CTA 0 alone)
    int own;          // points in a CTA's memory (of a slab at most)
    int u, b, r;      // byte offsets in shared memory: solution, right-hand side, residual (a split level's
                      // solution and residual have a halo row above and below)
    int a;            // and systems: pairs (h0, h1) [own], pairs (h2, det) [own], inv [own]
    int down, up;     // and row taps of the restriction to the next level / the prolongation to this one
    int team;         // threads of CTA 0 that run a whole level
    int near;         // a split level: every row a CTA's transfers read is one of its own or next to them
    Weights<T> w, g;  // relaxation weights (mem_weights) and operator weights (reg_weights)
};

template <typename T>
struct ResidentCycle {
    ResidentLevel<T> lv[kMaxLevels];
    int first, local, last;  // levels first .. local - 1 are split over the cluster, local .. last run on CTA 0
    int nit, cycles;
    int lgsize;              // log2 of the cluster's CTAs
    int silent;              // a CTA that sends no edge rows (-1: none; the self-test of the waits)
    unsigned long long timeout_ns;  // of an exchange's wait
    csg::Control* ctl;       // status word
};

// The start of a CTA's shared memory; the levels' fields and the row taps follow.  What
// follows addresses them by 32-bit byte offsets from the shared array itself: through pointers
// every access would need 64-bit address arithmetic or go through the generic address window.
// The plan is read from the kernel's parameters, which makes its values uniform to the
// compiler: a half-sweep is ~60 instructions of one chain, and every branch that might
// diverge adds 20-40 cycles to it (227 cycles with none, 440 with five).  So inner branches
// are on uniform values, and what depends on the lane is computed by all and stored under a
// predicate.
struct ResidentHead {
    alignas(8) unsigned long long barriers[2];
    int lost;
};
constexpr int kHead = 32;
static_assert(sizeof(ResidentHead) <= kHead);

extern __shared__ __align__(16) unsigned char resident_smem[];
__device__ __forceinline__ ResidentHead& resident_head() { return *reinterpret_cast<ResidentHead*>(resident_smem); }
template <typename T>
__device__ __forceinline__ Pair<T>& pair_at(int offset) {
    return *reinterpret_cast<Pair<T>*>(resident_smem + offset);
}
template <typename T>
__device__ __forceinline__ const AxisTaps<T>& taps_at(int offset, int k) {
    return *reinterpret_cast<const AxisTaps<T>*>(resident_smem + offset + k * static_cast<int>(sizeof(AxisTaps<T>)));
}
template <typename T>
__device__ __forceinline__ PointSystem<T> load_system(int a, int own, int i) {
    constexpr int kPair = sizeof(Pair<T>);
    const Pair<T> p = pair_at<T>(a + i * kPair), q = pair_at<T>(a + (own + i) * kPair);
    T inv = T(0);
    if constexpr (sizeof(T) == 8) inv = *reinterpret_cast<const T*>(resident_smem + a + 2 * own * kPair + i * sizeof(T));
    return {p.x, p.y, q.x, q.y, inv};
}
template <typename T>
__device__ __forceinline__ void store_system(int a, int own, int i, const PointSystem<T>& s) {
    constexpr int kPair = sizeof(Pair<T>);
    pair_at<T>(a + i * kPair) = {s.h0, s.h1};
    pair_at<T>(a + (own + i) * kPair) = {s.h2, s.det};
    if constexpr (sizeof(T) == 8) *reinterpret_cast<T*>(resident_smem + a + 2 * own * kPair + i * sizeof(T)) = s.inv;
}

// Every field of a level is an image of rows of nx pairs, a row holding its points of colour 0
// ((x + y) even) by ascending x, then those of colour 1: the points of one colour that the
// lanes of a warp hold, and each kind of neighbour of theirs, are consecutive in shared memory.
__device__ __forceinline__ int image_column(int y, int x, int nx) { return ((x + y) & 1) * (nx >> 1) + (x >> 1); }

// A point a thread holds in registers: its system and right-hand side.
template <typename T>
struct Point {
    PointSystem<T> s;
    Pair<T> b;
};

// The points (2 j, y) and (2 j + 1, y), one of each colour, as byte offsets in the image of u whose
// row y starts at `row`; each is the other's x neighbour on one side.  nx = 1: the row's one
// point, its own x neighbour.  At the image's top and bottom the y neighbour is the point itself.
struct Unit {
    int q[2];              // the points of colour 0 and 1
    int side[2];           // their other x neighbours
    int above[2], below[2];
    bool odd;              // the point of colour 0 is (2 j + 1, y)
};
template <typename T>
__device__ __forceinline__ Unit make_unit(int row, int y, int j, int nx, bool top, bool bottom) {
    constexpr int kPair = sizeof(Pair<T>);
    const int h = nx >> 1, next = j + 1 >= h ? 0 : j + 1, previous = j > 0 ? j - 1 : max(h - 1, 0);
    Unit m;
    m.odd = (y & 1) != 0 && nx > 1;
    m.q[0] = row + j * kPair;
    m.q[1] = m.q[0] + h * kPair;
    m.side[0] = row + (h + (m.odd ? next : previous)) * kPair;
    m.side[1] = row + (m.odd ? previous : next) * kPair;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        m.above[c] = top ? m.q[c] : m.q[1 - c] - nx * kPair;
        m.below[c] = bottom ? m.q[c] : m.q[1 - c] + nx * kPair;
    }
    return m;
}

// Sums of the y and of the x neighbours of a unit's point.
template <int COLOUR, typename T>
__device__ __forceinline__ void neighbour_sums(const Unit& m, Pair<T>& ys, Pair<T>& xs) {
    const Pair<T> a = pair_at<T>(m.above[COLOUR]), b = pair_at<T>(m.below[COLOUR]);
    const Pair<T> c = pair_at<T>(m.q[1 - COLOUR]), d = pair_at<T>(m.side[COLOUR]);
    ys = {a.x + b.x, a.y + b.y};
    xs = {c.x + d.x, c.y + d.y};
}

// relax_core at a held point.
template <int COLOUR, typename T>
__device__ __forceinline__ Pair<T> relaxed(const Unit& m, const Point<T>& p, const Weights<T>& w) {
    Pair<T> ys, xs;
    neighbour_sums<COLOUR>(m, ys, xs);
    const T rx = p.b.x - w.w01 * ys.x - w.w10 * xs.x;
    const T ry = p.b.y - w.w01 * ys.y - w.w10 * xs.y;
    const T dxx = p.s.h0 + w.w00, dyy = p.s.h1 + w.w00;
    return quotients(dyy * rx - p.s.h2 * ry, -p.s.h2 * rx + dxx * ry, p.s);
}

// membrane_apply_at's residual at a held point (w: the operator weights).
template <int COLOUR, typename T>
__device__ __forceinline__ Pair<T> residual(const Unit& m, const Point<T>& p, const Weights<T>& w) {
    Pair<T> ys, xs;
    neighbour_sums<COLOUR>(m, ys, xs);
    const Pair<T> v = pair_at<T>(m.q[COLOUR]);
    const T reg0 = w.w00 * v.x + w.w01 * ys.x + w.w10 * xs.x;
    const T reg1 = w.w00 * v.y + w.w01 * ys.y + w.w10 * xs.y;
    return {p.b.x - (reg0 + p.s.h0 * v.x + p.s.h2 * v.y), p.b.y - (reg1 + p.s.h2 * v.x + p.s.h1 * v.y)};
}

// ---- transfers between levels whose x sizes are powers of two: resize_value of both
// components, the inner sums down the three source rows first.  The column weights are exact
// values of col_taps.  Halving reads columns 2 X .. 2 X + 2, doubling x / 2 - 1 .. x / 2 + 1 by the
// parity of x; between levels of one column it is that column three times.

template <typename T>
__device__ __forceinline__ void add_row(Pair<T> (&v)[3], int r, T w, const Pair<T>& p0, const Pair<T>& p1, const Pair<T>& p2) {
    const Pair<T> p[3] = {p0, p1, p2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const Pair<T> d{w * p[k].x, w * p[k].y};
        v[k] = r == 0 ? d : Pair<T>{v[k].x + d.x, v[k].y + d.y};
    }
}
template <typename T>
__device__ __forceinline__ Pair<T> column_sum(const Pair<T> (&v)[3], T w0, T w1, T w2) {
    return {w0 * v[0].x + w1 * v[1].x + w2 * v[2].x, w0 * v[0].y + w1 * v[1].y + w2 * v[2].y};
}
template <typename T>
__device__ __forceinline__ Pair<T> halved(const Pair<T> (&v)[3], bool same) {
    return column_sum<T>(v, same ? T(0.125) : T(0.5), same ? T(0.75) : T(0.5), same ? T(0.125) : T(0));
}
template <typename T>
__device__ __forceinline__ Pair<T> doubled(const Pair<T> (&v)[3], bool same, bool odd) {
    return column_sum<T>(v, same ? T(0.125) : (odd ? T(0.03125) : T(0.28125)), same ? T(0.75) : T(0.6875),
                         same ? T(0.125) : (odd ? T(0.28125) : T(0.03125)));
}
// The sums down the rows t.o of the image at byte offset f (its row `lo` first) of columns x - 1,
// x, x + 1 (periodic).
template <typename T>
__device__ __forceinline__ void row_sums(int f, int lo, const AxisTaps<T>& t, int x, int nx, Pair<T> (&v)[3]) {
    constexpr int kPair = sizeof(Pair<T>);
    const int half = (nx >> 1) * kPair, mask = nx - 1;
    const int before = (((x - 1) & mask) >> 1) * kPair, centre = (x >> 1) * kPair, after = (((x + 1) & mask) >> 1) * kPair;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int g = t.o[r], row = f + (g - lo) * nx * kPair, shift = ((x + g) & 1) * half;
        const int own = row + shift, other = row + half - shift;
        add_row(v, r, t.w[r], pair_at<T>(other + before), pair_at<T>(own + centre), pair_at<T>(other + after));
    }
}

// ---- levels of CTA 0.  A thread holds one unit.  A level's team is as many threads as it has
// units, rounded up to 32, 64 or 256; a smaller team synchronises in fewer cycles.

// (a branch by team to __syncwarp or an immediate barrier costs 30 cycles more)
__device__ __forceinline__ void team_sync(int id, int team) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(team) : "memory");
}
__device__ __forceinline__ int team_barrier(int team) { return team == 32 ? 1 : team == 64 ? 2 : 4; }

// One visit of a level of CTA 0 in a V-cycle by its team.  up: prolongation of level
// l + 1's solution, then relaxation.  Else relaxation and, unless l is the last level, the
// residual and its restriction to level l + 1, whose solution is zeroed.
template <typename T>
__device__ __forceinline__ void local_visit(const ResidentCycle<T>& c, int l, bool up) {
    constexpr int kPair = sizeof(Pair<T>);
    const ResidentLevel<T>& L = c.lv[l];
    const ResidentLevel<T>& N = c.lv[l + 1 <= c.last ? l + 1 : l];
    const int nx = L.nx, ny = L.ny, team = L.team, id = team_barrier(team), h = nx >> 1, thread = threadIdx.x;
    const int row = thread >> (L.lg > 0 ? L.lg - 1 : 0), j = h > 0 ? thread & (h - 1) : 0;
    const bool same = nx == 1, in = row < ny;
    const int y = in ? row : ny - 1;  // (a thread without a unit computes the last row's again)
    const bool has0 = in && (!same || (y & 1) == 0), has1 = in && (!same || (y & 1) != 0);
    const int u = L.u, i = y * nx + j;
    const Unit m = make_unit<T>(u + y * nx * kPair, y, j, nx, y == 0, y == ny - 1);
    const Point<T> p0{load_system<T>(L.a, L.own, i), pair_at<T>(L.b + i * kPair)};
    const Point<T> p1{load_system<T>(L.a, L.own, i + h), pair_at<T>(L.b + (i + h) * kPair)};
    if (up) {
        Pair<T> v[3];
        row_sums(N.u, 0, taps_at<T>(L.up, y), j, N.nx, v);
        const Pair<T> d0 = doubled(v, same, m.odd), d1 = doubled(v, same, !m.odd), v0 = pair_at<T>(m.q[0]),
                      v1 = pair_at<T>(m.q[1]);
        if (in) pair_at<T>(m.q[0]) = {v0.x + d0.x, v0.y + d0.y};
        if (in && !same) pair_at<T>(m.q[1]) = {v1.x + d1.x, v1.y + d1.y};
        team_sync(id, team);
    }
    const Weights<T> w = L.w;
    const int nit = c.nit;
#pragma unroll 1
    for (int it = 0; it < nit; ++it) {
        const Pair<T> v1 = relaxed<1>(m, p1, w);
        if (has1) pair_at<T>(m.q[1]) = v1;
        team_sync(id, team);
        const Pair<T> v0 = relaxed<0>(m, p0, w);
        if (has0) pair_at<T>(m.q[0]) = v0;
        team_sync(id, team);
    }
    if (up || l == c.last) return;
    const int r = L.r - u;
    const Weights<T> g = L.g;
    const Pair<T> r1 = residual<1>(m, p1, g), r0 = residual<0>(m, p0, g);
    if (has1) pair_at<T>(m.q[1] + r) = r1;
    if (has0) pair_at<T>(m.q[0] + r) = r0;
    team_sync(id, team);
    const int snx = N.nx;
    for (int k = thread; k < N.own; k += team) {
        const int X = k & (snx - 1), Y = k >> N.lg;
        Pair<T> v[3];
        row_sums(L.r, 0, taps_at<T>(L.down, Y), same ? 0 : 2 * X + 1, nx, v);
        pair_at<T>(N.b + (Y * snx + image_column(Y, X, snx)) * kPair) = halved(v, same);
        pair_at<T>(N.u + k * kPair) = Pair<T>{T(0), T(0)};
    }
    team_sync(id, team);
}

// The V-cycle's levels local .. last on CTA 0; a thread takes part while the level's team includes
// it, and on the way up waits for the smaller team of the level below.
template <typename T>
__device__ __forceinline__ void local_cycle(const ResidentCycle<T>& c) {
    const int thread = threadIdx.x, local = c.local, last = c.last;
    // (visits in one uniform sequence, down then up)
    const int visits = 2 * (last - local) + 1;
#pragma unroll 1
    for (int k = 0; k < visits; ++k) {
        const bool up = k > last - local;
        const int l = up ? 2 * last - local - k : local + k, team = c.lv[l].team;
        if (thread >= team) continue;
        if (up && c.lv[l + 1].team != team) team_sync(team_barrier(team), team);  // the smaller team is done with l + 1
        local_visit<T>(c, l, up);
    }
    __syncthreads();
}

// ---- levels split over the cluster

__device__ __forceinline__ unsigned shared_address(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// The address, in the cluster's shared window, of byte offset `offset` of CTA `rank`'s shared memory.
__device__ __forceinline__ unsigned cluster_address(int offset, int rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(shared_address(resident_smem + offset)), "r"(rank));
    return a;
}
// Where `on`, store a pair in another CTA's shared memory and count its bytes on a barrier there.
__device__ __forceinline__ void send(bool on, unsigned to, unsigned barrier, const Pair<double>& v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%1], {%2, %3}, [%4];\n\t}" ::"r"(static_cast<unsigned>(on)),
                 "r"(to), "l"(__double_as_longlong(v.x)), "l"(__double_as_longlong(v.y)), "r"(barrier)
                 : "memory");
}
__device__ __forceinline__ void send(bool on, unsigned to, unsigned barrier, const Pair<float>& v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%1], {%2, %3}, [%4];\n\t}" ::"r"(static_cast<unsigned>(on)),
                 "r"(to), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(barrier)
                 : "memory");
}
// Plain stores (where `on`) and loads of another CTA's shared memory; cluster barriers order them.
__device__ __forceinline__ void put(bool on, unsigned to, const Pair<double>& v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared::cluster.v2.f64 [%1], {%2, %3};\n\t}" ::"r"(static_cast<unsigned>(on)),
                 "r"(to), "d"(v.x), "d"(v.y)
                 : "memory");
}
__device__ __forceinline__ void put(bool on, unsigned to, const Pair<float>& v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared::cluster.v2.f32 [%1], {%2, %3};\n\t}" ::"r"(static_cast<unsigned>(on)),
                 "r"(to), "f"(v.x), "f"(v.y)
                 : "memory");
}
__device__ __forceinline__ void get(unsigned from, Pair<double>& v) {
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(from) : "memory");
}
__device__ __forceinline__ void get(unsigned from, Pair<float>& v) {
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(from) : "memory");
}

// The edge-row exchange of the half-sweeps.  Half-sweep e sends each updated edge point to
// the neighbour's halo, counted on the neighbour's barrier e & 1, which completes when
// both neighbours' bytes have come and this CTA has announced them.  Half-sweep e waits for
// half-sweep e - 1.  Two barriers do, and a halo point is never overwritten before it is read: an
// edge unit reads its halo before it sends, and a neighbour starts its half-sweep e + 1, whose
// points of the halo this CTA's half-sweep e reads, only when all of this CTA's edge points
// of half-sweep e have been counted there.  An exchange of 16 CTAs in a chain takes 434 cycles from wait
// to wait.  (A cluster barrier with its release and acquire takes 570, 770-980 with remote stores before
// it; remote stores with one remote arrival per warp 1,120; bulk copies of the rows 470-480.)
//
// Every wait is bounded.  A thread whose wait runs out (or that sees another's run out) counts as
// lost from then on: it announces and sends nothing more, so no barrier's phase is announced twice and no
// neighbour's completes with rows that were not updated, but it goes on through every barrier of its CTA
// and cluster.  The first to give up tells all CTAs of the cluster; the whole grid's result becomes NaN and
// the status word CSG_ERR_TIMEOUT.
__device__ __forceinline__ bool exchanged(unsigned at, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(at), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __noinline__ bool await_exchange_slowly(unsigned at, unsigned parity, int* lost, int lgsize,
                                                   unsigned long long timeout_ns) {
    const unsigned long long start = csg::global_timer_ns();
    while (true) {
        if (*reinterpret_cast<volatile int*>(lost)) return false;
        if (exchanged(at, parity)) return true;
        if (csg::global_timer_ns() - start <= timeout_ns) continue;
        const unsigned mine = static_cast<unsigned>(__cvta_generic_to_shared(lost));
        for (int r = 0; r < 1 << lgsize; ++r)
            asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.u32 [a], 1;\n\t}" ::"r"(mine),
                         "r"(r)
                         : "memory");
        return false;
    }
}

// A CTA's rows of a split level.
struct Slab {
    int lo, n;  // its rows
    int lg, nx, ny;
    int rank, lgsize;
    __device__ __forceinline__ Slab(int lg_, int nx_, int ny_, int rank_, int lgsize_)
        : lg(lg_), nx(nx_), ny(ny_), rank(rank_), lgsize(lgsize_) {
        lo = begin(rank);
        n = begin(rank + 1) - lo;
    }
    __device__ __forceinline__ int begin(int r) const { return (r * ny) >> lgsize; }
    __device__ __forceinline__ bool above() const { return rank > 0; }
    __device__ __forceinline__ bool below() const { return rank + 1 < (1 << lgsize); }
};
template <typename T>
__device__ __forceinline__ Slab slab_of(const ResidentCycle<T>& c, int l) {
    return Slab(c.lv[l].lg, c.lv[l].nx, c.lv[l].ny, static_cast<int>(blockIdx.x), c.lgsize);
}

// row_sums over a field at byte offset f whose CTAs hold their rows between two halo rows.  near: the
// three rows are the CTA's own or its halo rows, else each is read from the CTA that holds it.
template <typename T>
__device__ __forceinline__ void slab_sums(const Slab& V, int f, bool near, const AxisTaps<T>& t, int x, Pair<T> (&v)[3]) {
    if (near) {
        row_sums(f, V.lo - 1, t, x, V.nx, v);
        return;
    }
#pragma unroll 1
    for (int r = 0; r < 3; ++r) {
        const int g = t.o[r];
        int owner = V.rank;
        while (g < V.begin(owner)) --owner;
        while (g >= V.begin(owner + 1)) ++owner;
        const unsigned row = cluster_address(f, owner) + (((g - V.begin(owner) + 1) << V.lg)) * static_cast<unsigned>(sizeof(Pair<T>));
        Pair<T> p[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            get(row + image_column(g, (x - 1 + k) & (V.nx - 1), V.nx) * static_cast<unsigned>(sizeof(Pair<T>)), p[k]);
        add_row(v, r, t.w[r], p[0], p[1], p[2]);
    }
}

// Two consecutive elements, in one read when the field is aligned for it.
template <typename T>
__device__ __forceinline__ Pair<T> load_two(const T* p, bool aligned) {
    if (aligned) return *reinterpret_cast<const Pair<T>*>(p);
    return {p[0], p[1]};
}

// The units of a CTA's first and last row come first: their points are sent early in a half-sweep and
// arrive while the others are updated.
__device__ __forceinline__ int unit_row(int k, int n) { return k == 0 ? 0 : (k == 1 ? n - 1 : k - 1); }

// One visit of a split level in a V-cycle.  up: prolongation of level l + 1's solution and
// relaxation; down: relaxation, the residual and its restriction to level l + 1, whose
// solution is zeroed.  Both: the end of one cycle and the start of the next on the first
// level, whose systems stay in registers in between.  A thread holds up to kResidentSlots
// units; e: iterations exchanged before; kept: none of the thread's waits has run out.
template <typename T>
__device__ __forceinline__ void split_visit(const ResidentCycle<T>& c, int l, int e, bool up, bool down, bool& kept) {
    constexpr int kPair = sizeof(Pair<T>);
    ResidentHead& S = resident_head();
    const ResidentLevel<T>& L = c.lv[l];
    const ResidentLevel<T>& N = c.lv[l + 1];
    const Slab V = slab_of<T>(c, l), W = slab_of<T>(c, l + 1);
    const int nx = V.nx, lg = V.lg, h = nx >> 1, thread = threadIdx.x, rank = V.rank, u = L.u;
    const bool whole = N.rows == 0, near = L.near != 0;
    // the thread's units; the first level's systems come from global memory
    const int count = V.n << (lg - 1);
    const int active = min(kResidentThreads, (count + 31) & ~31);  // threads with units, rounded to warps
    const int slots = (count + kResidentThreads - 1) / kResidentThreads;
    Unit m[kResidentSlots];
    Point<T> p[2][kResidentSlots];
    bool in[kResidentSlots], top[kResidentSlots], bottom[kResidentSlots];  // a unit in the slot; in the first, the last own
                                                                           // row with a CTA beyond it
#pragma unroll
    for (int s = 0; s < kResidentSlots; ++s) {
        if (s >= slots) break;
        int k = thread + s * kResidentThreads;
        in[s] = k < count;
        k = min(k, count - 1);  // (a thread without a unit computes the last one's again)
        const int row = unit_row(k >> (lg - 1), V.n), j = k & (h - 1);
        m[s] = make_unit<T>(u + ((row + 1) << lg) * kPair, V.lo + row, j, nx, V.lo + row == 0, V.lo + row == V.ny - 1);
        top[s] = in[s] && row == 0 && V.above() && rank != c.silent;
        bottom[s] = in[s] && row == V.n - 1 && V.below() && rank != c.silent;
        if (l == c.first) {
            const int P = nx * V.ny, at = ((V.lo + row) << lg) + 2 * j;
            const T* A = L.A + 3 * static_cast<size_t>(blockIdx.y) * P;
            const T* B = L.B + 2 * static_cast<size_t>(blockIdx.y) * P;
            const bool wide = ((reinterpret_cast<size_t>(A) | reinterpret_cast<size_t>(B)) & (2 * sizeof(T) - 1)) == 0;
            A += at;
            B += at;
            const Pair<T> h0 = load_two(A, wide), h1 = load_two(A + P, wide), h2 = load_two(A + 2 * P, wide);
            const Pair<T> bx = load_two(B, wide), by = load_two(B + P, wide);
            const bool odd = m[s].odd;
            p[0][s] = {point_system(odd ? h0.y : h0.x, odd ? h1.y : h1.x, odd ? h2.y : h2.x, L.w.w00),
                       {odd ? bx.y : bx.x, odd ? by.y : by.x}};
            p[1][s] = {point_system(odd ? h0.x : h0.y, odd ? h1.x : h1.y, odd ? h2.x : h2.y, L.w.w00),
                       {odd ? bx.x : bx.y, odd ? by.x : by.y}};
        } else {
            const int i = (row << lg) + j;
            p[0][s] = {load_system<T>(L.a, L.own, i), pair_at<T>(L.b + i * kPair)};
            p[1][s] = {load_system<T>(L.a, L.own, i + h), pair_at<T>(L.b + (i + h) * kPair)};
        }
    }
    // offset of the halo row of the CTA above that copies the first own row, minus that row's here;
    // the same for the last own row and the CTA below
    const unsigned above = (V.above() ? cluster_address(0, rank - 1) : 0) + (V.lo - V.begin(rank - 1)) * nx * kPair;
    const unsigned below = (V.below() ? cluster_address(0, rank + 1) : 0) - V.n * nx * kPair;
    if (up) {
        if (whole) {
            // CTA 0's solution: this CTA's rows need its rows lowest .. highest
            if (rank > 0) {
                const unsigned source = cluster_address(N.u, 0);
                const int lowest = taps_at<T>(L.up, 0).o[0] << N.lg, highest = (taps_at<T>(L.up, V.n - 1).o[2] + 1) << N.lg;
                for (int i = lowest + thread; i < highest; i += kResidentThreads)
                    get(source + i * kPair, pair_at<T>(N.u + i * kPair));
            }
            __syncthreads();
        }
#pragma unroll
        for (int s = 0; s < kResidentSlots; ++s) {
            if (s >= slots) break;
            const int k = min(thread + s * kResidentThreads, count - 1);
            const int row = unit_row(k >> (lg - 1), V.n), j = k & (h - 1);
            Pair<T> v[3];
            if (whole) row_sums(N.u, 0, taps_at<T>(L.up, row), j, N.nx, v);
            else slab_sums(W, N.u, near, taps_at<T>(L.up, row), j, v);
#pragma unroll
            for (int colour = 0; colour < 2; ++colour) {
                const int q = m[s].q[colour];
                const Pair<T> d = doubled(v, false, m[s].odd == (colour == 0)), b = pair_at<T>(q), z{b.x + d.x, b.y + d.y};
                if (in[s]) pair_at<T>(q) = z;
                put(top[s], above + q, z);
                put(bottom[s], below + q, z);
            }
        }
        cooperative_groups::this_cluster().sync();
    }
    if (thread < active) {
        // the half-sweeps of colour 1 use barrier 0, those of colour 0 barrier 1
        const unsigned barrier = shared_address(S.barriers);
        const int bytes = nx * static_cast<int>(sizeof(T)) * ((V.above() ? 1 : 0) + (V.below() ? 1 : 0));
        unsigned above_barrier = 0, below_barrier = 0;
        if (V.above()) above_barrier = cluster_address(0, rank - 1);
        if (V.below()) below_barrier = cluster_address(0, rank + 1);
        const Weights<T> w = L.w;
        const int end = e + c.nit * ((up ? 1 : 0) + (down ? 1 : 0));
        auto await_exchange = [&](unsigned at, int parity) {
            if (!exchanged(at, parity)) kept &= await_exchange_slowly(at, parity, &S.lost, c.lgsize, c.timeout_ns);
        };
        auto half_sweep = [&](auto colour_) {
            constexpr int colour = decltype(colour_)::value, mine = colour ? 0 : 8, theirs = 8 - mine;
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %0, 0;\n\t"
                "@p mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%1], %2;\n\t}" ::"r"(kept ? thread : 1),
                "r"(barrier + mine), "r"(bytes)
                : "memory");
            await_exchange(barrier + theirs, (colour ? e - 1 : e) & 1);
#pragma unroll
            for (int s = 0; s < kResidentSlots; ++s) {
                if (s >= slots) break;
                // (as if h0 and h1 changed: the sums h + w00 of eight points would not fit the registers)
                if constexpr (sizeof(T) == 8) asm volatile("" : "+d"(p[colour][s].s.h0), "+d"(p[colour][s].s.h1));
                const int q = m[s].q[colour];
                const Pair<T> v = relaxed<colour>(m[s], p[colour][s], w);
                if (in[s]) pair_at<T>(q) = v;
                if (s * kResidentThreads < nx) {  // the units of the first and the last row
                    send(top[s] && kept, above + q, above_barrier + mine, v);
                    send(bottom[s] && kept, below + q, below_barrier + mine, v);
                }
            }
            asm volatile("bar.sync 3, %0;" ::"r"(active) : "memory");
        };
#pragma unroll 1
        for (; e < end; ++e) {
            half_sweep(std::integral_constant<int, 1>{});
            half_sweep(std::integral_constant<int, 0>{});
        }
        await_exchange(barrier + 8, (e - 1) & 1);
        if (down) {
            const Weights<T> g = L.g;
            const int r = L.r - u;
#pragma unroll
            for (int s = 0; s < kResidentSlots; ++s) {
                if (s >= slots) break;
#pragma unroll
                for (int colour = 0; colour < 2; ++colour) {
                    const int q = m[s].q[colour] + r;
                    const Pair<T> z = colour ? residual<1>(m[s], p[1][s], g) : residual<0>(m[s], p[0][s], g);
                    if (in[s]) pair_at<T>(q) = z;
                    if (s * kResidentThreads < nx) {
                        put(top[s], above + q, z);
                        put(bottom[s], below + q, z);
                    }
                }
            }
        }
    }
    if (!down) {
        // the next prolongation reads this CTA's rows and halo rows only, unless they are not near
        if (l > c.first && c.lv[l - 1].near != 0) __syncthreads();
        else cooperative_groups::this_cluster().sync();
        return;
    }
    // the next level's solution starts from zero (a neighbour writes its halo rows only after the barrier)
    if (!whole || rank == 0) {
        const int n = whole ? N.own : (N.rows + 2) << N.lg;
        for (int i = thread; i < n; i += kResidentThreads) pair_at<T>(N.u + i * kPair) = Pair<T>{T(0), T(0)};
    }
    cooperative_groups::this_cluster().sync();
    const unsigned home = whole ? cluster_address(N.b + (W.lo << N.lg) * kPair, 0) : 0;  // the rows of a whole level go to CTA 0
    for (int i = thread; i < (W.n << N.lg); i += kResidentThreads) {
        const int X = i & (N.nx - 1), row = i >> N.lg, at = (row * N.nx + image_column(W.lo + row, X, N.nx)) * kPair;
        Pair<T> v[3];
        slab_sums(V, L.r, near, taps_at<T>(L.down, row), 2 * X + 1, v);
        if (whole) put(true, home + at, halved(v, false));
        else pair_at<T>(N.b + at) = halved(v, false);
    }
    if (whole || !near) cooperative_groups::this_cluster().sync();
    else __syncthreads();
}

// c.cycles V-cycles from level c.first on, one cluster per batch element (blockIdx.y).
template <typename T, int CTAS>
__global__ void __launch_bounds__(kResidentThreads, CTAS) k_resident_cycles(const __grid_constant__ ResidentCycle<T> c) {
    constexpr int kPair = sizeof(Pair<T>);
    csg::pdl_begin();
    ResidentHead& S = resident_head();
    const int rank = blockIdx.x;  // the grid's x dimension is one cluster
    const size_t bi = blockIdx.y;
    const bool split = c.local > c.first;
    if (threadIdx.x == 0) {
        S.lost = 0;
        const unsigned barrier = shared_address(S.barriers);
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barrier) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barrier + 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // The fields and tables of all levels, each as one list over the levels with several loads in
    // flight per thread: level by level every one waits for its loads in turn (4 us more per launch).
    constexpr int kAhead = 4;
    const int thread = threadIdx.x;
    // the row's points of level l that this CTA holds systems for in shared memory (the first split
    // level's are read when it is visited) and its first one
    auto held = [&](int l, int& lo) {
        const ResidentLevel<T>& L = c.lv[l];
        const Slab V(L.lg, L.nx, L.ny, rank, c.lgsize);
        lo = L.rows > 0 ? V.lo : 0;
        return L.rows > 0 ? (l > c.first ? V.n << L.lg : 0) : (rank == 0 ? L.nx * L.ny : 0);
    };
    int points = 0, lo;
    for (int l = c.first; l <= c.last; ++l) points += held(l, lo);
    for (int k0 = thread; k0 < points; k0 += kAhead * kResidentThreads) {
        T h[kAhead][3];
        int level[kAhead], at[kAhead];
#pragma unroll
        for (int s = 0; s < kAhead; ++s) {
            int k = k0 + s * kResidentThreads, l = c.first;
            level[s] = -1;
            if (k >= points) continue;
            for (int n = held(l, lo); k >= n; n = held(++l, lo)) k -= n;
            const ResidentLevel<T>& L = c.lv[l];
            const int P = L.nx * L.ny, row = k >> L.lg;
            const T* A = L.A + 3 * bi * P + (lo << L.lg) + k;
            level[s] = l;
            at[s] = (row << L.lg) + image_column(lo + row, k & (L.nx - 1), L.nx);
            h[s][0] = __ldg(A);
            h[s][1] = __ldg(A + P);
            h[s][2] = __ldg(A + 2 * P);
        }
#pragma unroll
        for (int s = 0; s < kAhead; ++s)
            if (level[s] >= 0) {
                const ResidentLevel<T>& L = c.lv[level[s]];
                store_system(L.a, L.own, at[s], point_system(h[s][0], h[s][1], h[s][2], L.w.w00));
            }
    }
    {
        // the first level's u, with its halo rows when it is split (rows outside the grid are never
        // read), and b when it is not
        const ResidentLevel<T>& L = c.lv[c.first];
        const Slab V(L.lg, L.nx, L.ny, rank, c.lgsize);
        const int P = L.nx * L.ny, halo = split ? 1 : 0, total = (V.n + 2 * halo) << L.lg;
        const T* U = L.U + 2 * bi * P;
        const T* B = L.B + 2 * bi * P;
        for (int j0 = thread; j0 < total; j0 += 2 * kAhead * kResidentThreads) {
            Pair<T> v[2 * kAhead];
#pragma unroll
            for (int s = 0; s < 2 * kAhead; ++s) {
                const int j = j0 + s * kResidentThreads, g = V.lo - halo + (j >> L.lg), i = (g << L.lg) + (j & (L.nx - 1));
                if (j < total && g >= 0 && g < L.ny) v[s] = Pair<T>{U[i], U[P + i]};
            }
#pragma unroll
            for (int s = 0; s < 2 * kAhead; ++s) {
                const int j = j0 + s * kResidentThreads, row = j >> L.lg, g = V.lo - halo + row;
                const int q = ((row << L.lg) + image_column(g, j & (L.nx - 1), L.nx)) * kPair;
                if (j < total && g >= 0 && g < L.ny) pair_at<T>(L.u + q) = v[s];
            }
        }
        if (!split)
            for (int i = thread; i < P; i += kResidentThreads) {
                const int y = i >> L.lg;
                pair_at<T>(L.b + ((y << L.lg) + image_column(y, i & (L.nx - 1), L.nx)) * kPair) = Pair<T>{B[i], B[P + i]};
            }
    }
    // row taps (row numbers and weights) of the rows this CTA restricts to and prolongates to
    for (int k = thread, l = c.first, base = 0; l < c.last;) {
        const ResidentLevel<T>& L = c.lv[l];
        const ResidentLevel<T>& N = c.lv[l + 1];
        const bool whole = L.rows == 0;
        const Slab V(L.lg, L.nx, L.ny, rank, c.lgsize), W(N.lg, N.nx, N.ny, rank, c.lgsize);
        const int nn = whole ? N.ny : W.n, n = whole ? L.ny : V.n, i = k - base;
        if (i >= nn + n) {
            base += nn + n;
            ++l;
            continue;
        }
        const bool down = i < nn;
        const int row = down ? (whole ? 0 : W.lo) + i : (whole ? 0 : V.lo) + i - nn;
        AxisTaps<T>* taps = reinterpret_cast<AxisTaps<T>*>(resident_smem + (down ? L.down : L.up));
        taps[down ? i : i - nn] = row_taps<T>(row, down ? L.ny : N.ny, down ? N.ny : L.ny, 1);
        k += kResidentThreads;
    }
    if (split) cooperative_groups::this_cluster().sync();
    else __syncthreads();
    // Down the split levels, the levels of CTA 0, up again; on the first level the end of a cycle
    // and the start of the next are one visit.  (One call of each visit, as they are inlined:
    // behind a call every half-sweep takes 160 cycles more.)
    int e = 0, l = c.first, cycle = 0;  // e: iterations exchanged
    bool up = false, kept = true;
#pragma unroll 1
    while (true) {
        if (l == c.local) {
            if (rank == 0) local_cycle<T>(c);
            if (!split) {
                if (++cycle == c.cycles) break;
                continue;
            }
            cooperative_groups::this_cluster().sync();
            up = true;
            --l;
        }
        if (l == c.first && up) ++cycle;
        const bool down = !up || (l == c.first && cycle < c.cycles);
        split_visit<T>(c, l, e, up, down, kept);
        e += c.nit * ((up ? 1 : 0) + (down ? 1 : 0));
        if (l == c.first && cycle == c.cycles) break;
        if (down) {
            up = false;
            ++l;
        } else {
            --l;
        }
    }
    const ResidentLevel<T>& F = c.lv[c.first];
    const int P = F.nx * F.ny, halo = split ? 1 : 0;
    T* U = F.U + 2 * bi * P;
    // The cluster has met after its last exchange: no CTA stores to another's memory past here, and all agree on
    // whether a wait ran out.  If none did, every exchange has been waited for.
    const bool lost = *reinterpret_cast<volatile int*>(&S.lost) != 0;
    const Slab V(F.lg, F.nx, F.ny, rank, c.lgsize);
    for (int i = threadIdx.x; i < V.n << F.lg; i += kResidentThreads) {
        const int row = i >> F.lg;
        const Pair<T> v =
            pair_at<T>(F.u + (((row + halo) << F.lg) + image_column(V.lo + row, i & (F.nx - 1), F.nx)) * kPair);
        U[(V.lo << F.lg) + i] = lost ? T(NAN) : v.x;
        U[P + (V.lo << F.lg) + i] = lost ? T(NAN) : v.y;
    }
    if (lost) {
        if (rank == 0 && threadIdx.x == 0 && atomicCAS(&c.ctl->status, CSG_OK, CSG_ERR_TIMEOUT) == CSG_OK)
            c.ctl->where = static_cast<int>(bi);
        // edge points sent before the last barrier may still be on their way to this CTA: a millisecond outlasts them
        const unsigned long long start = csg::global_timer_ns();
        while (csg::global_timer_ns() - start < 1000000ull) {
        }
    }
}

// ------------------------------------------------ V-cycle legs of the levels above
//
// A level too fine for a resident V-cycle takes one launch down (2 nit half-sweeps, the
// residual and its restriction) and one up (the prolongation and 2 nit half-sweeps): a CTA
// holds a tile and a halo, runs the leg's steps on them and writes back its tile.  A
// half-sweep reads only neighbours one step away, so after k of them the values are exact
// at least k cells inside the region's cut edges; with a halo of 2 nit + 2 the tile and one
// ring round it hold exact residuals for the restriction taps (2 nit going up).  What lies
// outside is computed all the same, from whatever the region's wrapped rows give, and never used.
// The points are held as in a resident level -- systems and right-hand sides in registers,
// u in an image split by colour -- and see the operations of the separate kernels in their
// order, so results are bit-identical.
//
// Separate launches are bound by reading 56 bytes per point for each half-sweep from L2: on two
// 512 x 256 float64 grids 6.7 us each, 104 us a V-cycle for the level, where both legs take 52
// although they update each point 2.5 times.  A V-cycle of the whole hierarchy with three
// iterations: 171 -> 123 us (eight grids 353 -> 326, two in float32 154 -> 106, one of
// 1024 x 512 271 -> 190).  The halo grows with the iterations and a tile shrinks: a point is updated
// 2.8 times at four of them, 4 at five, 7 at six, 28 at eight (one 512 x 256 grid at eight: 403 us
// against 275, eight of them at five: 566 against 493), so the cheaper form is estimated
// for each launch (see LegCosts).

constexpr int kLegUnits = kResidentSlots * kResidentThreads;  // of a region, one row of tap weights each at most 128
constexpr int kLegWidth = 48;                                 // columns of a region (nx when fewer); 40-64 within 2%, 80 10% slower
constexpr int kLegRows = 128;                                 // rows at most

// A leg reads the level's solution from Uin and writes its tiles to Uout, a
// different buffer: tiles of one launch read each other's halos, so none may
// overwrite what another still reads (down: U -> the level's R buffer; up:
// R -> U).
template <typename T>
struct FineLeg {
    const T* A;    // this level's Hessian [batch][3][ny][nx]
    const T* B;    // right-hand side [batch][2][ny][nx]
    const T* Uin;  // solution before the leg [batch][2][ny][nx]
    T* Uout;       // solution after the leg
    T* nB;         // down: the next coarser level's right-hand side (restricted residual)
    T* nU;         // down: the next coarser level's solution (zeroed); up: the coarser solution to prolongate
    int nx, ny, cnx, cny;
    int width, halo, tw, th, tiles_x;  // region columns; tile size (tw = width = nx: whole rows)
    int nit;
    int wide;      // the fields are aligned for pairs of elements
    Weights<T> w, g;
};

template <typename T>
__device__ __forceinline__ void store_two(T* p, const Pair<T>& v, bool aligned) {
    if (aligned) {
        *reinterpret_cast<Pair<T>*>(p) = v;
    } else {
        p[0] = v.x;
        p[1] = v.y;
    }
}

template <typename T, bool DOWN>
__global__ void __launch_bounds__(kResidentThreads, sizeof(T) == 4 ? 2 : 1)
    k_vcycle_leg(const __grid_constant__ FineLeg<T> L) {
    constexpr int kPair = sizeof(Pair<T>);
    csg::pdl_begin();
    const int nx = L.nx, ny = L.ny, w = L.width, h = w >> 1, thread = threadIdx.x, P = nx * ny, cP = L.cnx * L.cny;
    const int tx = static_cast<int>(blockIdx.x) % L.tiles_x, ty = static_cast<int>(blockIdx.x) / L.tiles_x;
    const int x0 = tx * L.tw, x1 = min(nx, x0 + L.tw), y0 = ty * L.th, y1 = min(ny, y0 + L.th);
    const int gx0 = w == nx ? 0 : x0 - L.halo, gy0 = max(0, y0 - L.halo), wy = min(ny, y1 + L.halo) - gy0;
    const int count = h * wy, slots = (count + kResidentThreads - 1) / kResidentThreads;
    const bool wide = L.wide != 0;
    // shared memory: u, the residual (down), row taps
    const int u = 0, image = wy * w * kPair, taps = DOWN ? 2 * image : image;
    const size_t bi = blockIdx.y;
    const T* A = L.A + 3 * bi * P;
    const T* B = L.B + 2 * bi * P;
    const T* Uin = L.Uin + 2 * bi * P;
    // taps of the coarse rows whose centre tap may lie in the tile / of the region's rows
    // (64-bit products: they pass 2^31 from 65,536 rows on)
    const int Y0 = DOWN ? max(0, static_cast<int>((y0 - 2LL) * L.cny / ny) - 1) : gy0;
    const int rows = DOWN ? min(L.cny, static_cast<int>((y1 + 2LL) * L.cny / ny) + 2) - Y0 : wy;
    for (int k = thread; k < rows; k += kResidentThreads)
        reinterpret_cast<AxisTaps<T>*>(resident_smem + taps)[k] =
            DOWN ? row_taps<T>(Y0 + k, ny, L.cny, 1) : row_taps<T>(Y0 + k, L.cny, ny, L.cnx);
    if (!DOWN) __syncthreads();
    Unit m[kResidentSlots];
    Point<T> p[2][kResidentSlots];
    bool in[kResidentSlots];
#pragma unroll
    for (int s = 0; s < kResidentSlots; ++s) {
        if (s >= slots) break;
        int k = thread + s * kResidentThreads;
        in[s] = k < count;
        k = min(k, count - 1);  // (a thread without a unit computes the last one's again)
        const int row = k / h, j = k - row * h, gy = gy0 + row;
        int gx = gx0 + 2 * j;
        gx = gx < 0 ? gx + nx : (gx >= nx ? gx - nx : gx);
        const int at = gy * nx + gx;
        m[s] = make_unit<T>(u + row * w * kPair, gy, j, w, row == 0, row == wy - 1);
        const bool odd = m[s].odd;
        const Pair<T> h0 = load_two(A + at, wide), h1 = load_two(A + P + at, wide), h2 = load_two(A + 2 * P + at, wide);
        const Pair<T> bx = load_two(B + at, wide), by = load_two(B + P + at, wide);
        Pair<T> ux = load_two(Uin + at, wide), uy = load_two(Uin + P + at, wide);
        p[0][s] = {point_system(odd ? h0.y : h0.x, odd ? h1.y : h1.x, odd ? h2.y : h2.x, L.w.w00),
                   {odd ? bx.y : bx.x, odd ? by.y : by.x}};
        p[1][s] = {point_system(odd ? h0.x : h0.y, odd ? h1.x : h1.y, odd ? h2.x : h2.y, L.w.w00),
                   {odd ? bx.x : bx.y, odd ? by.x : by.y}};
        if (!DOWN) {
            const AxisTaps<T> t = taps_at<T>(taps, row);
            const T* f = L.nU + 2 * bi * cP;
            const int c = gx >> 1, c0 = c > 0 ? c - 1 : L.cnx - 1, c2 = c + 1 < L.cnx ? c + 1 : 0;
            Pair<T> v[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const T* g = f + t.o[r];
                add_row(v, r, t.w[r], Pair<T>{g[c0], g[cP + c0]}, Pair<T>{g[c], g[cP + c]}, Pair<T>{g[c2], g[cP + c2]});
            }
            const Pair<T> even = doubled(v, false, false), other = doubled(v, false, true);
            ux = {ux.x + even.x, ux.y + other.x};
            uy = {uy.x + even.y, uy.y + other.y};
        }
        if (in[s]) {
            pair_at<T>(m[s].q[0]) = {odd ? ux.y : ux.x, odd ? uy.y : uy.x};
            pair_at<T>(m[s].q[1]) = {odd ? ux.x : ux.y, odd ? uy.x : uy.y};
        }
    }
    __syncthreads();
    auto half_sweep = [&](auto colour_) {
        constexpr int colour = decltype(colour_)::value;
#pragma unroll
        for (int s = 0; s < kResidentSlots; ++s) {
            if (s >= slots) break;
            if constexpr (sizeof(T) == 8) asm volatile("" : "+d"(p[colour][s].s.h0), "+d"(p[colour][s].s.h1));  // (see split_visit)
            const Pair<T> v = relaxed<colour>(m[s], p[colour][s], L.w);
            if (in[s]) pair_at<T>(m[s].q[colour]) = v;
        }
        __syncthreads();
    };
#pragma unroll 1
    for (int it = 0; it < L.nit; ++it) {
        half_sweep(std::integral_constant<int, 1>{});
        half_sweep(std::integral_constant<int, 0>{});
    }
    T* Uout = L.Uout + 2 * bi * P;
#pragma unroll
    for (int s = 0; s < kResidentSlots; ++s) {
        if (s >= slots) break;
        if (DOWN) {
            const Pair<T> r0 = residual<0>(m[s], p[0][s], L.g), r1 = residual<1>(m[s], p[1][s], L.g);
            if (in[s]) {
                pair_at<T>(m[s].q[0] + image) = r0;
                pair_at<T>(m[s].q[1] + image) = r1;
            }
        }
        const int k = thread + s * kResidentThreads, row = k / h, x = gx0 + 2 * (k - row * h), y = gy0 + row;
        if (k >= count || x < x0 || x >= x1 || y < y0 || y >= y1) continue;
        const bool odd = m[s].odd;
        const Pair<T> a = pair_at<T>(m[s].q[0]), b = pair_at<T>(m[s].q[1]);
        store_two(Uout + y * nx + x, Pair<T>{odd ? b.x : a.x, odd ? a.x : b.x}, wide);
        store_two(Uout + P + y * nx + x, Pair<T>{odd ? b.y : a.y, odd ? a.y : b.y}, wide);
    }
    if (!DOWN) return;
    __syncthreads();
    // restriction of the residual to the coarse points whose centre tap (2 X + 1, the row's) lies in this tile
    const int cw = (x1 - x0) >> 1;
    T* nB = L.nB + 2 * bi * cP;
    T* nU = L.nU + 2 * bi * cP;
    for (int k = thread; k < cw * rows; k += kResidentThreads) {
        const int Y = k / cw, j = ((x0 - gx0) >> 1) + k - Y * cw, after = j + 1 >= h ? 0 : j + 1;
        const AxisTaps<T> t = taps_at<T>(taps, Y);
        if (t.o[1] < y0 || t.o[1] >= y1) continue;  // another tile's coarse row
        Pair<T> v[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int row = image + (t.o[r] - gy0) * w * kPair, shift = (t.o[r] & 1) * h * kPair;
            add_row(v, r, t.w[r], pair_at<T>(row + shift + j * kPair), pair_at<T>(row + h * kPair - shift + j * kPair),
                    pair_at<T>(row + shift + after * kPair));
        }
        const Pair<T> z = halved(v, false);
        const int at = (Y0 + Y) * L.cnx + (x0 >> 1) + k - Y * cw;
        nB[at] = z.x;
        nB[cP + at] = z.y;
        nU[at] = T(0);
        nU[cP + at] = T(0);
    }
}

constexpr size_t kLegSmemMax = 200 * 1024;

// What a wave of clusters spends on a resident V-cycle, in microseconds, summed over its levels: on a split
// level split + split_nit x iterations, (unit + unit_nit x iterations) for each unit of a thread, far where its
// transfers read other CTAs' rows; on a level of CTA 0 local + local_nit x iterations.  Fitted to V-cycles
// of 32 x 17 to 256 x 128 points, batches of 2 to 4,096 and 1 to 5 iterations (5% off at most in float64, 8% with
// two CTAs to an SM, 23% with one in float32).  Clusters of 16 CTAs run 7 at a time, so a batch of 32 grids of
// 256 x 128 in float32 took three waves of 82 us, where legs on the first level and clusters of
// 4 CTAs below take 156 (64 in float64 551 and 483 us, 128 of 256 x 113 with one iteration 757 and
// 490, and 587 before there were resident cycles).  In one wave, and with one CTA per grid, the resident form is
// the faster one throughout.
struct ResidentCosts {
    double split, split_nit, unit, unit_nit, far, local, local_nit;
};
template <typename T>
constexpr ResidentCosts resident_costs(bool paired) {
    if (sizeof(T) == 8) return {2.1, 0.69, 2.0, 0.85, 1.0, 1.0, 0.58};
    if (paired) return {3.9, -1.86, 1.1, 2.9, 1.3, 0.84, 1.14};
    return {1.8, 0.79, 0.71, 1.2, 0.43, 0.70, 0.83};
}
// A resident launch in every cycle, below legs, against one for all cycles: each loads its fields again.
// The estimates are up to 20% off where neither form is far ahead, so only a clear gain counts.
constexpr double kRelaunch = 9.5, kClearly = 0.85;

// What one V-cycle spends on a level above the resident ones, in microseconds: as two legs, a
// wave of CTAs (148 at once, 296 in float32) takes leg + leg_nit x iterations; as separate
// launches, each of the 4 x iterations + 4 takes launch + point per 100,000 points.  Fitted to
// V-cycles of 16 x 4096 to 2048 x 1024 points, batches of 1 to 128 and 1 to 8 iterations in both forms
// (an estimated V-cycle is 8% off on average, 35% at most); where it picks the slower form, the two
// differ by less than 5%.
template <typename T>
struct LegCosts {
    static constexpr bool f64 = sizeof(T) == 8;
    static constexpr double leg = f64 ? 7.6 : 6.8, leg_nit = f64 ? 0.95 : 1.18;
    static constexpr double launch = f64 ? 3.3 : 3.4, point = f64 ? 1.0 : 0.74;
    static constexpr double resident = f64 ? 148 : 296;
};

constexpr size_t kResidentSmemMax = 226 * 1024;
constexpr size_t kPairedSmemMax = 113 * 1024;  // of each of two CTAs to an SM
// The restriction chain of a level-l field to every coarser level at or below
// kChainPoints points per grid, in one launch with one CTA per batch element:
// the same resize_at per point as separate k_resize launches, level after
// level, with __syncthreads between levels.  Each restricted level is kept in
// shared memory (at most ~700 points x channels over all levels) as the
// source of the next one, and written to its field.
constexpr int kChainThreads = 1024;
constexpr int kChainPoints = 512;  // measured: 512 beats 2,048 (7.96 vs 8.14 ms per 256 x 128 solve) and matches 128

template <typename T>
struct ResizeChain {
    T* field[kMaxLevels];  // [batch * channels][ny][nx] per level
    int nx[kMaxLevels], ny[kMaxLevels];
    int off[kMaxLevels];   // offset of level l's [channels][ny][nx] image in shared memory (elements)
    int first, last, channels;
};

template <typename T>
__global__ void __launch_bounds__(kChainThreads) k_resize_chain(ResizeChain<T> c) {
    csg::pdl_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* base = reinterpret_cast<T*>(smem_raw);
    const int bi = blockIdx.x;
    // every level's row and column taps first (after the level images), then the levels
    int words = 0, ntaps = 0;
    for (int l = c.first; l <= c.last; ++l) {
        words += c.channels * c.nx[l] * c.ny[l];
        ntaps += c.nx[l] + c.ny[l];
    }
    AxisTaps<T>* taps = reinterpret_cast<AxisTaps<T>*>(smem_raw + ((static_cast<size_t>(words) * sizeof(T) + 15) & ~size_t(15)));
    for (int l = c.first, at = 0; l <= c.last; ++l) {
        for (int k = threadIdx.x; k < c.ny[l] + c.nx[l]; k += blockDim.x)
            taps[at + k] = k < c.ny[l] ? row_taps<T>(k, c.ny[l - 1], c.ny[l], c.nx[l - 1])
                                       : col_taps<T>(k - c.ny[l], c.nx[l - 1], c.nx[l]);
        at += c.ny[l] + c.nx[l];
    }
    __syncthreads();
    for (int l = c.first, at = 0; l <= c.last; ++l) {
        const int P = c.nx[l] * c.ny[l];
        const size_t plane0 = static_cast<size_t>(c.channels) * bi;
        T* image = base + c.off[l];
        T* out = c.field[l] + plane0 * P;
        const T* src = l == c.first ? c.field[l - 1] + plane0 * c.nx[l - 1] * c.ny[l - 1] : base + c.off[l - 1];
        const AxisTaps<T>* rows = taps + at;
        const AxisTaps<T>* cols = rows + c.ny[l];
        for (int j = threadIdx.x; j < c.channels * P; j += blockDim.x) {
            const int ch = j / P, i = j - ch * P;
            const T r = resize_value(src + static_cast<size_t>(ch) * c.nx[l - 1] * c.ny[l - 1], rows[i / c.nx[l]],
                                     cols[i % c.nx[l]]);
            out[j] = r;
            image[j] = r;
        }
        at += c.ny[l] + c.nx[l];
        __syncthreads();
    }
}

template <typename T>
size_t resize_chain_smem(const ResizeChain<T>& c) {
    size_t words = 0, taps = 0;
    for (int l = c.first; l <= c.last; ++l) {
        words += static_cast<size_t>(c.channels) * c.nx[l] * c.ny[l];
        taps += static_cast<size_t>(c.nx[l] + c.ny[l]);
    }
    return ((words * sizeof(T) + 15) & ~size_t(15)) + taps * sizeof(AxisTaps<T>);
}

// Opt the leg, resident-cycle and chain kernels in to more than 48 KB of dynamic
// shared memory, once per type and device (the first solve on a device runs eagerly, before any capture).
template <typename T>
void allow_big_smem() {
    static std::atomic<unsigned long long> done{0};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return;
    const unsigned long long bit = 1ULL << device;
    if (done.load() & bit) return;
    for (const void* leg : {reinterpret_cast<const void*>(k_vcycle_leg<T, true>), reinterpret_cast<const void*>(k_vcycle_leg<T, false>)})
        cudaFuncSetAttribute(leg, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kLegSmemMax));
    for (const void* kernel : {reinterpret_cast<const void*>(k_resident_cycles<T, 1>),
                               reinterpret_cast<const void*>(k_resident_cycles<T, sizeof(T) == 4 ? 2 : 1>)}) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kResidentSmemMax));
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    cudaFuncSetAttribute(reinterpret_cast<const void*>(k_resize_chain<T>), cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(kLegSmemMax));
    done.fetch_or(bit);
}

// Clusters of 1, 2, 4, 8 and 16 CTAs of a resident kernel that this device runs at once: with kResidentSmemMax of
// shared memory per CTA (one CTA to an SM), and of the kernel of two CTAs to an SM with half of that.  0: a size
// that the device refuses.  Found once per device.
struct ClusterCounts {
    int one[5], two[5];
};
template <typename T>
ClusterCounts cluster_counts() {
    static std::atomic<int> known[64][10];
    ClusterCounts counts{};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return counts;
    allow_big_smem<T>();
    for (int k = 9; k >= 0; --k) {
        int found = known[device][k].load() - 1;
        if (found < 0) {
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = 1u << k % 5;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cudaLaunchConfig_t config{};
            config.gridDim = dim3(1u << k % 5, 1, 1);
            config.blockDim = dim3(kResidentThreads, 1, 1);
            config.dynamicSmemBytes = k < 5 ? kResidentSmemMax : kPairedSmemMax;
            config.attrs = &attr;
            config.numAttrs = 1;
            const void* kernel = k < 5 ? reinterpret_cast<const void*>(k_resident_cycles<T, 1>)
                                       : reinterpret_cast<const void*>(k_resident_cycles<T, sizeof(T) == 4 ? 2 : 1>);
            if (cudaOccupancyMaxActiveClusters(&found, kernel, &config) != cudaSuccess) {
                cudaGetLastError();  // a size the device refuses is not the caller's error
                found = 0;
            }
            known[device][k].store(found + 1);
        }
        (k < 5 ? counts.one[k] : counts.two[k - 5]) = found;
    }
    return counts;
}

template <typename T>
__global__ void k_sub(T* __restrict__ v, const T* __restrict__ u, size_t n) {
    csg::pdl_begin();
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) v[i] = v[i] - u[i];
}

template <typename T>
__global__ void k_any_nonzero(const T* __restrict__ u, size_t n, int* flag) {
    csg::pdl_begin();
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    // one plain store per CTA at most: every writer stores the same value (an atomic per
    // nonzero element took 14 us at 512 x 256, this 5)
    if (__syncthreads_or(i < n && u[i] != T(0)) && threadIdx.x == 0) *flag = 1;
}

// Fixed-order reduction of per-block partials into metrics[b * stride + slot]
// (objective = forward + reverse partials; reg * 0.5; sqrt(norm)), the blocks' partials
// added in block order.  The CTA stages a chunk of each of the four rows in shared memory
// and one thread of each of four warps adds a row from there: a thread reading global
// memory takes a round trip every few partials (512 x 256: 41 -> 9 us).
constexpr int kMetricsThreads = 256, kMetricsChunk = 512;

template <typename T>
__global__ void __launch_bounds__(kMetricsThreads) k_metrics(const T* __restrict__ obj_f, const T* __restrict__ obj_r,
                                                             const T* __restrict__ reg, const T* __restrict__ norm,
                                                             int nblocks, T* __restrict__ metrics, int metric_stride) {
    csg::pdl_begin();
    __shared__ T rows[4][kMetricsChunk];
    __shared__ T sums[4];
    const int b = blockIdx.x, row = threadIdx.x >> 5;
    const size_t at = static_cast<size_t>(b) * nblocks;
    const T* src[4] = {obj_f + at, obj_r ? obj_r + at : nullptr, reg + at, norm + at};
    T sum = T(0);
    for (int base = 0; base < nblocks; base += kMetricsChunk) {
        const int m = min(kMetricsChunk, nblocks - base);
        __syncthreads();
        for (int r = 0; r < 4; ++r)
            if (src[r])
                for (int i = threadIdx.x; i < m; i += blockDim.x) rows[r][i] = src[r][base + i];
        __syncthreads();
        if (row < 4 && (threadIdx.x & 31) == 0 && (row != 1 || obj_r)) {
            int i = 0;
            for (; i + 8 <= m; i += 8)
#pragma unroll
                for (int k = 0; k < 8; ++k) sum = sum + rows[row][i + k];
            for (; i < m; ++i) sum = sum + rows[row][i];
        }
    }
    if (row < 4 && (threadIdx.x & 31) == 0) sums[row] = sum;
    __syncthreads();
    if (threadIdx.x != 0) return;
    T* m = metrics + static_cast<size_t>(b) * metric_stride;
    m[0] = obj_r ? T(0.5) * sums[0] + T(0.5) * sums[1] : T(0.5) * sums[0];
    m[1] = sums[2] * T(0.5);
    m[2] = sqrt(sums[3]);
}

template <typename T>
__global__ void __launch_bounds__(csg::kOrderedThreads) k_objective_out(const T* __restrict__ partial, int nblocks,
                                                                         T* __restrict__ out) {
    csg::pdl_begin();
    __shared__ T buf[csg::kOrderedChunk];
    const T s = csg::ordered_sum(partial + static_cast<size_t>(blockIdx.x) * nblocks, nblocks, buf);
    if (threadIdx.x == 0) out[blockIdx.x] = T(0.5) * s;
}

// ------------------------------------------------------------- host side

struct Arena {
    char* base;
    size_t size;
    size_t used = 0;
    bool ok = true;
    template <typename T>
    T* take(size_t count) {
        const size_t bytes = (count * sizeof(T) + 255) & ~static_cast<size_t>(255);
        if (used + bytes > size) {
            ok = false;
            return nullptr;
        }
        T* p = reinterpret_cast<T*>(base ? base + used : nullptr);
        used += bytes;
        return p;
    }
};

inline dim3 grid_for(int points, int batch) { return dim3((points + kThreads - 1) / kThreads, batch); }

std::vector<std::pair<int, int>> grid_levels(int nx, int ny) {
    std::vector<std::pair<int, int>> specs{{nx, ny}};
    while (specs.back().first >= 2 || specs.back().second >= 2) {
        const auto prev = specs.back();
        const std::pair<int, int> coarse{(prev.first + 1) / 2, (prev.second + 1) / 2};
        specs.push_back(coarse);
        if (coarse.first < 2 && coarse.second < 2) break;
    }
    return specs;
}

bool relax_supported(int nx) { return nx % 2 == 0 || nx == 1; }

// Multigrid workspace for one (batch, nx, ny).
template <typename T>
struct FmgBuffers {
    std::vector<std::pair<int, int>> specs;
    std::vector<T*> A, B, B0, U, R;
    csg::Control* ctl = nullptr;  // the scratch's first 256 bytes: status word, and the flag of k_any_nonzero
    int* flag = nullptr;
    void take_control(Arena& ar) {
        ctl = ar.take<csg::Control>(1);
        flag = ctl ? ctl->pad : nullptr;
    }
    bool carve(Arena& ar, int batch, int nx, int ny) {
        specs = grid_levels(nx, ny);
        const size_t L = specs.size();
        A.assign(L, nullptr);
        B.assign(L, nullptr);
        B0.assign(L, nullptr);
        U.assign(L, nullptr);
        R.assign(L, nullptr);
        for (size_t l = 0; l < L; ++l) {
            const size_t P = static_cast<size_t>(specs[l].first) * specs[l].second;
            if (l > 0) {
                A[l] = ar.take<T>(3 * P * batch);
                B[l] = ar.take<T>(2 * P * batch);
                B0[l] = ar.take<T>(2 * P * batch);
                U[l] = ar.take<T>(2 * P * batch);
            }
            R[l] = ar.take<T>(2 * P * batch);
        }
        return ar.ok;
    }
};

template <typename T>
struct Fmg {
    FmgBuffers<T>& buf;
    int batch;
    double base[5];
    int cycles, nit;
    cudaStream_t s;
    int nx0, ny0;
    double timeout_s = 2.0;
    int silent = -1;

    void params_at(size_t l, double out[5]) const {
        out[0] = base[0] * buf.specs[l].first / nx0;
        out[1] = base[1] * buf.specs[l].second / ny0;
        out[2] = base[2];
        out[3] = base[3];
        out[4] = base[4];
    }
    void relax(size_t l) {
        const int nx = buf.specs[l].first, ny = buf.specs[l].second;
        double pr[5];
        params_at(l, pr);
        const MemWeights w = mem_weights(pr);
        for (int it = 0; it < 2 * nit; ++it)
            (csg::note_launch(), csg::launch_pdl(k_relax<T>, grid_for(nx * ny, batch), kThreads, 0, s, buf.A[l], buf.B[l], buf.U[l], nx, ny,
                                                                      it % 2 == 0 ? 1 : 0, T(w.w00), T(w.w01), T(w.w10)));
    }
    void resize(const T* src, size_t from, T* dst, size_t to, int channels, bool accumulate) {
        const auto f = buf.specs[from], t = buf.specs[to];
        (csg::note_launch(), csg::launch_pdl(k_resize<T>, grid_for(t.first * t.second, batch * channels), kThreads, 0, s, src, dst, f.first, f.second,
                                                                                     t.first, t.second, accumulate));
    }
    // The resident launch of `count` V-cycles from level `first` on, or size 0 when the level
    // does not fit one cluster: more than kResidentPoints points for a CTA of it (256 x 128
    // fits 16 CTAs, 512 x 256 does not), too much shared memory, or an x size that is no power of
    // two.  A cluster has a CTA per kCoarsePoints points and no more CTAs than any split level has rows.
    struct Resident {
        ResidentCycle<T> c{};
        int size = 0;
        size_t smem = 0;
        bool paired = false;  // two CTAs to an SM
        int waves = 1;
        double us = 0;        // estimated time of a V-cycle
    };
    Resident resident(size_t first, int count) const {
        Resident none, plan;
        const size_t L = buf.specs.size();
        if (L > static_cast<size_t>(kMaxLevels) || nit < 1) return none;
        const ClusterCounts counts = cluster_counts<T>();
        auto points = [&](size_t l) { return static_cast<long long>(buf.specs[l].first) * buf.specs[l].second; };
        size_t local = first;
        while (points(local) > kCoarsePoints) ++local;  // the last level is one point
        int size = 1;
        if (local > first) {
            int most = 1;
            for (int k = 1; k < 5; ++k)
                if (counts.one[k] > 0) most = 1 << k;
            while (size < most && points(first) > static_cast<long long>(size) * kCoarsePoints) size *= 2;
            for (size_t l = first; l < local; ++l) {
                if (buf.specs[l].first < 2) return none;
                while (buf.specs[l].second < size) size /= 2;
            }
            while (size > 2 && static_cast<long long>(size) * batch > kPairedCtas &&
                   2 * points(first) <= static_cast<long long>(size) * kResidentPoints)
                size /= 2;
            if (size < 2) return none;
        }
        ResidentCycle<T>& c = plan.c;
        c.first = static_cast<int>(first);
        c.local = static_cast<int>(local);
        c.last = static_cast<int>(L - 1);
        c.nit = nit;
        c.cycles = count;
        c.silent = silent;
        c.timeout_ns = static_cast<unsigned long long>(timeout_s * 1e9);
        c.ctl = buf.ctl;
        while ((1 << c.lgsize) < size) ++c.lgsize;
        long long at = kHead;
        auto take = [&](long long elements) {  // a byte offset of that many elements, aligned for pairs
            const long long here = at;
            at += (elements * static_cast<long long>(sizeof(T)) + 15) / 16 * 16;
            return static_cast<int>(here);
        };
        int residual = 0;
        for (size_t l = first; l < L; ++l) {
            double pr[5];
            params_at(l, pr);
            const MemWeights w = mem_weights(pr);
            const RegWeights g = reg_weights(pr, 1);
            ResidentLevel<T>& V = c.lv[l];
            V.A = buf.A[l];
            V.B = buf.B[l];
            V.U = buf.U[l];
            V.nx = buf.specs[l].first;
            V.ny = buf.specs[l].second;
            while ((1 << V.lg) < V.nx) ++V.lg;
            if ((1 << V.lg) != V.nx) return none;
            const bool split = l < local;
            V.rows = split ? (V.ny + size - 1) / size : 0;
            const long long own = split ? static_cast<long long>(V.rows) * V.nx : points(l);
            if (split && own > kResidentPoints) return none;
            V.own = static_cast<int>(own);
            if (l == first && split) residual = take(2 * (own + 2LL * V.nx));
            V.u = take(split ? 2 * (own + 2LL * V.nx) : 2 * own);
            V.b = l == first && split ? 0 : take(2 * own);
            V.r = split ? residual : take(2 * own);
            V.a = l == first && split ? 0 : take((sizeof(T) == 8 ? 5 : 4) * own);
            const int units = V.ny * std::max(1, V.nx / 2);
            if (!split && units > kResidentThreads) return none;  // (a level one point wide)
            V.team = units > 64 ? kResidentThreads : units > 32 ? 64 : 32;
            V.w = {T(w.w00), T(w.w01), T(w.w10)};
            V.g = {T(g.w[0]), T(g.w[1]), T(g.w[2])};
            if (l + 1 < L) {
                const int ny1 = buf.specs[l + 1].second;
                const int kTaps = static_cast<int>(sizeof(AxisTaps<T>) / sizeof(T));
                V.near = split && V.ny == 2 * ny1 && ny1 % size == 0;
                V.down = take(kTaps * (split ? (ny1 + size - 1) / size : ny1));
                V.up = take(kTaps * (split ? V.rows : V.ny));
            }
        }
        if (at > kResidentSmemMax) return none;
        plan.smem = static_cast<size_t>(at);
        plan.size = size;
        plan.paired = sizeof(T) == 4 && static_cast<long long>(size) * batch > kPairedCtas;
        const int at_once = std::max(1, (plan.paired && plan.smem <= kPairedSmemMax ? counts.two : counts.one)[c.lgsize]);
        plan.waves = (batch + at_once - 1) / at_once;
        const ResidentCosts k = resident_costs<T>(plan.paired);
        for (int l = c.first; l < c.local; ++l) {
            const int units = (c.lv[l].own / 2 + kResidentThreads - 1) / kResidentThreads;  // of a thread
            plan.us += k.split + k.split_nit * nit + (k.unit + k.unit_nit * nit) * units + (c.lv[l].near ? 0.0 : k.far);
        }
        plan.us = plan.waves * (plan.us + (c.last - c.local + 1) * (k.local + k.local_nit * nit));
        return plan;
    }
    void launch_resident(const Resident& plan) {
        allow_big_smem<T>();
        auto kernel = k_resident_cycles<T, 1>;
        if (plan.paired) kernel = k_resident_cycles<T, sizeof(T) == 4 ? 2 : 1>;
        (csg::note_launch(), csg::launch_pdl_cluster(kernel, dim3(static_cast<unsigned>(plan.size), static_cast<unsigned>(batch)),
                                                     static_cast<unsigned>(plan.size), kResidentThreads, plan.smem, s, plan.c));
    }
    // The leg of level l, where it can run as one: an even x size, and halos that leave some of a
    // region's columns and rows (of 48 x 42 up to nit = 9).
    bool leg(size_t l, bool down, const T* uin, T* uout, FineLeg<T>& g) const {
        const int nx = buf.specs[l].first, ny = buf.specs[l].second;
        if (nx % 2 != 0 || nit < 1 || nit > 64) return false;
        g = FineLeg<T>{};
        g.halo = 2 * nit + (down ? 2 : 0);
        g.width = std::min(nx, kLegWidth);
        const int rows = std::min(ny, std::min(kLegRows, 2 * kLegUnits / g.width));
        g.tw = g.width == nx ? nx : g.width - 2 * g.halo;
        g.th = rows == ny ? ny : rows - 2 * g.halo;
        if (g.tw < 2 || g.th < 2) return false;
        g.tiles_x = (nx + g.tw - 1) / g.tw;
        double pr[5];
        params_at(l, pr);
        const MemWeights w = mem_weights(pr);
        const RegWeights r = reg_weights(pr, 1);
        g.w = {T(w.w00), T(w.w01), T(w.w10)};
        g.g = {T(r.w[0]), T(r.w[1]), T(r.w[2])};
        g.A = buf.A[l];
        g.B = buf.B[l];
        g.Uin = uin;
        g.Uout = uout;
        g.nx = nx;
        g.ny = ny;
        g.nB = buf.B[l + 1];
        g.nU = buf.U[l + 1];
        g.cnx = buf.specs[l + 1].first;
        g.cny = buf.specs[l + 1].second;
        g.nit = nit;
        g.wide = ((reinterpret_cast<size_t>(g.A) | reinterpret_cast<size_t>(g.B) | reinterpret_cast<size_t>(uin) |
                   reinterpret_cast<size_t>(uout)) %
                  (2 * sizeof(T))) == 0;
        return true;
    }
    static int leg_tiles(const FineLeg<T>& g) { return g.tiles_x * ((g.ny + g.th - 1) / g.th); }
    // Whether level l runs as legs, by the estimate of LegCosts, and its time.
    bool as_legs(size_t l, double& us) const {
        using C = LegCosts<T>;
        const double points = static_cast<double>(buf.specs[l].first) * buf.specs[l].second * batch;
        us = (4.0 * nit + 4.0) * (C::launch + C::point * 1e-5 * points);
        FineLeg<T> down, up;
        if (!leg(l, true, buf.U[l], buf.R[l], down) || !leg(l, false, buf.R[l], buf.U[l], up)) return false;
        const double waves = std::max(1.0, leg_tiles(down) * static_cast<double>(batch) / C::resident) +
                             std::max(1.0, leg_tiles(up) * static_cast<double>(batch) / C::resident);
        const double legs = waves * (C::leg + C::leg_nit * nit);
        if (legs > us) return false;
        us = legs;
        return true;
    }
    template <bool DOWN>
    void launch_leg(const FineLeg<T>& g) {
        allow_big_smem<T>();
        const int rows = std::min(g.ny, g.th == g.ny ? g.ny : g.th + 2 * g.halo);
        const size_t smem = static_cast<size_t>(rows) * g.width * sizeof(Pair<T>) * (DOWN ? 2 : 1) +
                            (rows + 8) * sizeof(AxisTaps<T>);
        const dim3 grid(static_cast<unsigned>(leg_tiles(g)), static_cast<unsigned>(batch));
        (csg::note_launch(), csg::launch_pdl(k_vcycle_leg<T, DOWN>, grid, kResidentThreads, smem, s, g));
    }
    // `count` V-cycles from level `start` on: the levels above the resident ones as legs or separate
    // launches in every cycle.  Resident from the first level that fits a cluster, unless the batch takes
    // several waves of clusters and a later level is estimated to be faster (see ResidentCosts).
    void run_cycles(size_t start, int count) {
        if (count < 1) return;
        const size_t last = buf.specs.size() - 1;
        size_t fit = last;
        Resident plan;
        std::vector<char> legs;  // whether level start + i runs as legs
        double above = 0;        // estimated time of the levels before l
        for (size_t l = start; plan.size == 0 || above < plan.us; ++l) {
            Resident r = resident(l, l == start ? count : 1);
            if (r.size > 0) {
                if (l > start) r.us += above + kRelaunch;
                if (plan.size == 0 || r.us < kClearly * plan.us) {
                    plan = r;
                    fit = l;
                }
                if (r.waves == 1 || r.size == 1) break;
            }
            if (l == last) break;
            double us = 0;
            legs.push_back(as_legs(l, us));
            above += us;
        }
        if (plan.size > 0 && fit == start) {
            launch_resident(plan);
            return;
        }
        FineLeg<T> g;
        for (int c = 0; c < count; ++c) {
            // down: relax, residual, restriction (a fused leg leaves the relaxed solution in R[l]);
            // up: prolongation, relax (a fused leg reads R[l] and writes U[l])
            for (size_t l = start; l < fit; ++l) {
                const int nx = buf.specs[l].first, ny = buf.specs[l].second;
                if (legs[l - start] && leg(l, true, buf.U[l], buf.R[l], g)) {
                    launch_leg<true>(g);
                    continue;
                }
                relax(l);
                double pr[5];
                params_at(l, pr);
                (csg::note_launch(), csg::launch_pdl(k_membrane_apply<T>, grid_for(nx * ny, batch), kThreads, 0, s,
                                                     buf.A[l], buf.U[l], buf.B[l], buf.R[l], nx, ny, reg_weights(pr, 1)));
                resize(buf.R[l], l, buf.B[l + 1], l + 1, 2, false);
                const size_t P1 = static_cast<size_t>(buf.specs[l + 1].first) * buf.specs[l + 1].second;
                cudaMemsetAsync(buf.U[l + 1], 0, 2 * P1 * batch * sizeof(T), s);
            }
            if (plan.size > 0) launch_resident(plan);
            else relax(last);
            for (size_t l = fit; l-- > start;) {
                if (legs[l - start] && leg(l, false, buf.R[l], buf.U[l], g)) {
                    launch_leg<false>(g);
                    continue;
                }
                resize(buf.U[l + 1], l + 1, buf.U[l], l, 2, true);
                relax(l);
            }
        }
    }
    // Solves into buf.U[0]; U[0] must already hold the initial guess (or
    // zeros when `coarse_init`).  hess / rhs are level-0 A / B.
    // A[l] = resize(A[l - 1]) for every level: separate launches down to
    // kChainPoints points per grid, then the rest in one k_resize_chain launch.
    void restrict_hessians() {
        const size_t L = buf.specs.size();
        size_t l = 1;
        for (; l < L && static_cast<long long>(buf.specs[l].first) * buf.specs[l].second > kChainPoints; ++l)
            resize(buf.A[l - 1], l - 1, buf.A[l], l, 3, false);
        if (l >= L) return;
        if (L > static_cast<size_t>(kMaxLevels)) {
            for (; l < L; ++l) resize(buf.A[l - 1], l - 1, buf.A[l], l, 3, false);
            return;
        }
        ResizeChain<T> c{};
        for (size_t k = 0; k < L; ++k) {
            c.field[k] = buf.A[k];
            c.nx[k] = buf.specs[k].first;
            c.ny[k] = buf.specs[k].second;
        }
        c.first = static_cast<int>(l);
        c.last = static_cast<int>(L - 1);
        c.channels = 3;
        for (int k = c.first, off = 0; k <= c.last; ++k) {
            c.off[k] = off;
            off += c.channels * c.nx[k] * c.ny[k];
        }
        allow_big_smem<T>();
        (csg::note_launch(), csg::launch_pdl(k_resize_chain<T>, batch, kChainThreads, resize_chain_smem(c), s, c));
    }
    void run(bool coarse_init) {
        const size_t L = buf.specs.size();
        restrict_hessians();
        if (!coarse_init) {
            // every V-cycle writes each coarser level's right-hand side and zeroes its
            // solution before reading them, so the warm start needs no clearing
            run_cycles(0, cycles);
            return;
        }
        for (size_t l = 1; l < L; ++l) resize(l == 1 ? buf.B[0] : buf.B0[l - 1], l - 1, buf.B0[l], l, 2, false);
        for (size_t l = 1; l < L; ++l) {
            const size_t P = static_cast<size_t>(buf.specs[l].first) * buf.specs[l].second;
            cudaMemsetAsync(buf.B[l], 0, 2 * P * batch * sizeof(T), s);
            cudaMemsetAsync(buf.U[l], 0, 2 * P * batch * sizeof(T), s);
        }
        const size_t last = L - 1;
        const size_t Pl = static_cast<size_t>(buf.specs[last].first) * buf.specs[last].second;
        (csg::note_launch(), csg::launch_pdl(k_point_solve<T>, grid_for(static_cast<int>(Pl), batch), kThreads, 0, s, 
            buf.A[last], last == 0 ? buf.B[0] : buf.B0[last], buf.U[last], static_cast<int>(Pl), T(base[4])));
        relax(last);
        for (size_t l = last; l-- > 0;) {
            resize(buf.U[l + 1], l + 1, buf.U[l], l, 2, false);
            if (l > 0) {
                const size_t P = static_cast<size_t>(buf.specs[l].first) * buf.specs[l].second;
                cudaMemcpyAsync(buf.B[l], buf.B0[l], 2 * P * batch * sizeof(T), cudaMemcpyDeviceToDevice, s);
            }
            run_cycles(l, cycles);
        }
    }
};

// Workspace of one dartel_step for a batch.
template <typename T>
struct StepBuffers {
    T *map[2], *jac[2], *smap[2], *sjac[2], *rmap[2], *rjac[2];
    T *rhs_f[2], *hess_f[2], *rhs_r[2], *hess_r[2];
    T *rhs, *hess, *objf, *objr, *preg, *pnorm;
    FmgBuffers<T> fmg;
    int nblocks;
    bool carve(Arena& ar, int batch, int nx, int ny) {
        const size_t P = static_cast<size_t>(nx) * ny * batch;
        fmg.take_control(ar);
        for (int i = 0; i < 2; ++i) {
            map[i] = ar.take<T>(2 * P);
            jac[i] = ar.take<T>(4 * P);
            smap[i] = ar.take<T>(2 * P);
            sjac[i] = ar.take<T>(4 * P);
            rmap[i] = ar.take<T>(2 * P);
            rjac[i] = ar.take<T>(4 * P);
            rhs_f[i] = ar.take<T>(2 * P);
            hess_f[i] = ar.take<T>(3 * P);
            rhs_r[i] = ar.take<T>(2 * P);
            hess_r[i] = ar.take<T>(3 * P);
        }
        nblocks = (nx * ny + kThreads - 1) / kThreads;
        objf = ar.take<T>(static_cast<size_t>(nblocks) * batch);
        objr = ar.take<T>(static_cast<size_t>(nblocks) * batch);
        preg = ar.take<T>(static_cast<size_t>(nblocks) * batch);
        pnorm = ar.take<T>(static_cast<size_t>(nblocks) * batch);
        // rhs / hess of the solve live in the multigrid's level-0 slots
        if (!fmg.carve(ar, batch, nx, ny)) return false;
        rhs = ar.take<T>(2 * P);
        hess = ar.take<T>(3 * P);
        return ar.ok;
    }
};

// squaring_update (dartel_grid.py:778-914) with the reference's two-slot
// bookkeeping: slot `other` receives each step's b increment and, when the
// map is composed, the composed map; slot 0 after the loop is the
// "scratch" dartel_step hands to the multigrid as its initial guess.
// Returns the index of the current slot; b / a end in rb[cur_ba] / ha[cur_ba].
template <typename T>
struct Squaring {
    int cur_map, cur_ba;
};

template <typename T>
Squaring<T> run_squaring(T* rb[2], T* ha[2], T* maps[2], T* jacs[2], int k, bool save, int batch, int nx, int ny,
                         cudaStream_t s) {
    const dim3 g = grid_for(nx * ny, batch);
    int cur = 0, other = 1, ba = 0;
    for (int step = 0; step < k; ++step) {
        if (save || step < k - 1) {
            (csg::note_launch(), csg::launch_pdl(k_squaring_compose<T>, g, kThreads, 0, s, rb[ba], ha[ba], maps[cur],
                                                 jacs[cur], rb[1 - ba], ha[1 - ba], maps[other], jacs[other], nx, ny));
            std::swap(cur, other);
        } else {
            (csg::note_launch(), csg::launch_pdl(k_squaring<T>, g, kThreads, 0, s, rb[ba], ha[ba], maps[cur], jacs[cur],
                                                 rb[1 - ba], ha[1 - ba], maps[other], nx, ny));
        }
        ba = 1 - ba;
    }
    if (save && cur != 0) {
        const size_t P = static_cast<size_t>(nx) * ny * batch;
        cudaMemcpyAsync(maps[0], maps[cur], 2 * P * sizeof(T), cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(jacs[0], jacs[cur], 4 * P * sizeof(T), cudaMemcpyDeviceToDevice, s);
    }
    return {cur, ba};
}

template <typename T>
int dartel_step_impl(StepBuffers<T>& W, const T* source, const T* target, T* velocity, T* metrics, int metric_stride,
                     int batch, int nx, int ny, int k, const double* params, double lmreg, int cycles, int nit,
                     int code, int assume_initial_nonzero, bool first, cudaStream_t s) {
    if (first) CSG_CUDA_CHECK(cudaMemsetAsync(W.fmg.ctl, 0, sizeof(csg::Control), s));
    const dim3 g = grid_for(nx * ny, batch);
    const double scale = 1.0 / static_cast<double>(1LL << k);
    const size_t P = static_cast<size_t>(nx) * ny * batch;
    // expdef(v, k) with Jacobian
    (csg::note_launch(), csg::launch_pdl(k_smalldef<T>, g, kThreads, 0, s, velocity, W.map[0], W.jac[0], nx, ny, T(scale), T(scale * 0.5)));
    int cur = 0;
    for (int i = 0; i < k; ++i) {
        (csg::note_launch(), csg::launch_pdl(k_compose<T>, g, kThreads, 0, s, W.map[cur], W.jac[cur], W.map[cur], W.jac[cur], W.map[1 - cur],
                                            W.jac[1 - cur], nx, ny));
        cur = 1 - cur;
    }
    // forward objective with jac_div_smalldef(J, v, s)
    (csg::note_launch(), csg::launch_pdl(k_objfun<T, true>, g, kThreads, 0, s, source, target, W.map[cur], W.jac[cur], velocity, nullptr, W.rhs_f[0],
                                             W.hess_f[0], W.objf, nx, ny, T(scale * 0.5)));
    // squaring of the forward terms from smalldef_jac(v, -s)
    (csg::note_launch(), csg::launch_pdl(k_smalldef<T>, g, kThreads, 0, s, velocity, W.smap[0], W.sjac[0], nx, ny, T(-scale), T(-scale * 0.5)));
    Squaring<T> fw = run_squaring<T>(W.rhs_f, W.hess_f, W.smap, W.sjac, k, code == 1, batch, nx, ny, s);
    T* initial = W.smap[0];
    T* rr = nullptr;
    T* hr = nullptr;
    if (code == 1) {
        (csg::note_launch(), csg::launch_pdl(k_objfun<T, true>, g, kThreads, 0, s, target, source, W.smap[fw.cur_map], W.sjac[fw.cur_map], velocity,
                                                 nullptr, W.rhs_r[0], W.hess_r[0], W.objr, nx, ny, T(-scale * 0.5)));
        (csg::note_launch(), csg::launch_pdl(k_smalldef<T>, g, kThreads, 0, s, velocity, W.rmap[0], W.rjac[0], nx, ny, T(scale), T(scale * 0.5)));
        Squaring<T> rv = run_squaring<T>(W.rhs_r, W.hess_r, W.rmap, W.rjac, k, false, batch, nx, ny, s);
        initial = W.rmap[0];
        rr = W.rhs_r[rv.cur_ba];
        hr = W.hess_r[rv.cur_ba];
    }
    const RegWeights rw = reg_weights(params, 1);
    T* rhs = W.rhs;
    (csg::note_launch(), csg::launch_pdl(k_combine<T>, g, kThreads, 0, s, W.rhs_f[fw.cur_ba], rr, W.hess_f[fw.cur_ba], hr, velocity, rhs, W.hess, W.preg,
                                        W.pnorm, nx, ny, T(scale), rw));
    (csg::note_launch(), csg::launch_pdl(k_metrics<T>, batch, kMetricsThreads, 0, s, W.objf, code == 1 ? W.objr : nullptr, W.preg, W.pnorm, W.nblocks, metrics,
                                      metric_stride));
    // multigrid solve of (H + L) u = rhs from the scratch initial guess
    double solver[5] = {params[0], params[1], params[2], params[3], params[4] + lmreg};
    Fmg<T> fmg{W.fmg, batch, {solver[0], solver[1], solver[2], solver[3], solver[4]}, cycles, nit, s, nx, ny};
    W.fmg.A[0] = W.hess;
    W.fmg.B[0] = rhs;
    W.fmg.U[0] = initial;
    bool coarse_init = false;
    if (!assume_initial_nonzero) {
        csg::Control ctl{};
        if (!first) CSG_CUDA_CHECK(cudaMemsetAsync(W.fmg.flag, 0, sizeof(int), s));
        (csg::note_launch(), csg::launch_pdl(k_any_nonzero<T>, static_cast<unsigned>((2 * P + kThreads - 1) / kThreads), kThreads, 0, s, initial, 2 * P,
                                                                                                     W.fmg.flag));
        CSG_CUDA_CHECK(cudaMemcpyAsync(&ctl, W.fmg.ctl, offsetof(csg::Control, pad) + sizeof(int), cudaMemcpyDeviceToHost, s));
        CSG_CUDA_CHECK(cudaStreamSynchronize(s));
        if (ctl.status != CSG_OK)  // of an earlier step's solve
            return csg::fail(ctl.status, "dartel: a wait of the multigrid ran out (map %d)", ctl.where);
        coarse_init = ctl.pad[0] == 0;
        if (coarse_init) CSG_CUDA_CHECK(cudaMemsetAsync(initial, 0, 2 * P * sizeof(T), s));
    }
    fmg.run(coarse_init);
    (csg::note_launch(), csg::launch_pdl(k_sub<T>, static_cast<unsigned>((2 * P + kThreads - 1) / kThreads), kThreads, 0, s, velocity, initial, 2 * P));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

size_t dtype_size(int dtype) { return dtype == CSG_DTYPE_F64 ? 8 : 4; }

bool check_dtype(int dtype) { return dtype == CSG_DTYPE_F32 || dtype == CSG_DTYPE_F64; }

template <typename T>
size_t step_bytes(int batch, int nx, int ny) {
    Arena ar{nullptr, static_cast<size_t>(-1) / 2};
    StepBuffers<T> W;
    W.carve(ar, batch, nx, ny);
    return ar.used + 256;
}

template <typename T>
size_t expdef_bytes(int batch, int nx, int ny) {
    return 2 * (2 + 4) * static_cast<size_t>(nx) * ny * batch * sizeof(T) + 1024;
}

template <typename T>
int solve_typed(const void* source, const void* target, void* velocity, void* metrics, int batch, int nx,
                       int ny, int loop, const double* params, int its, double lmreg, int cycles, int nit, int code,
                       int assume, void* scratch, size_t bytes, cudaStream_t s) {
    Arena ar{static_cast<char*>(scratch), bytes};
    StepBuffers<T> W;
    if (!W.carve(ar, batch, nx, ny)) return csg::fail(CSG_ERR_ARG, "dartel: scratch of %zu bytes is too small", bytes);
    const int per = loop * its;
    for (int index = 0; index < loop; ++index)
        for (int it = 0; it < its; ++it) {
            int rc = dartel_step_impl<T>(W, static_cast<const T*>(source), static_cast<const T*>(target),
                                         static_cast<T*>(velocity), static_cast<T*>(metrics) + 3 * (index * its + it),
                                         3 * per, batch, nx, ny, index, params + 5 * index, lmreg, cycles, nit, code,
                                         assume, index == 0 && it == 0, s);
            if (rc) return rc;
        }
    return CSG_OK;
}

int check_grid(int dtype, int batch, int nx, int ny) {
    if (!check_dtype(dtype)) return csg::fail(CSG_ERR_ARG, "dartel: dtype must be CSG_DTYPE_F32 or CSG_DTYPE_F64");
    if (batch < 1 || nx < 1 || ny < 1) return csg::fail(CSG_ERR_ARG, "dartel: empty grid (%d x %d x %d)", batch, ny, nx);
    if (static_cast<long long>(nx) * ny > (1LL << 30)) return csg::fail(CSG_ERR_ARG, "dartel: grid too large");
    return CSG_OK;
}

// ------------------------------------------------ data-term adjoint
//
// E_b(v) = 1/2 sum_x (S_b(phi_k(x)) - T_b(x))^2 with phi_0 = id + v / 2^k and
// phi_{i+1} = phi_i o phi_i (the forward maps of expdef).  The adjoint runs
// the same bilinear stencils backwards: the sample step gives
// abar = r grad S(phi_k); each composition step C = F(A) with A = phi_i(x)
// and F = phi_i splits abar into the position part J_F(A)^T abar (added at
// x) and the value part (scattered to the four corner nodes with the
// bilinear weights, atomically).  The period unwrap of the corner values is
// a piecewise constant shift, so its derivative is the identity.

// Residual of one sample step, its block objective partial and (when abar is
// non-null) abar = r (dS/dX, dS/dY).
template <typename T>
__global__ void k_data_sample(const T* __restrict__ source, const T* __restrict__ target, const T* __restrict__ map,
                              T* __restrict__ abar, T* __restrict__ partial, int nx, int ny) {
    csg::pdl_begin();
    Pt p;
    const bool ok = point(nx, ny, p);
    T contrib = T(0);
    if (ok) {
        const int P = nx * ny;
        const size_t o1 = static_cast<size_t>(p.b) * P;
        const T* src = source + o1;
        const T* M = map + 2 * o1;
        const Stencil<T> st(M[p.i] - T(1), M[P + p.i] - T(1), nx, ny);
        const T k22 = src[st.i22], k12 = src[st.i12], k21 = src[st.i21], k11 = src[st.i11];
        const T sampled = (k22 * st.dx2 + k12 * st.dx1) * st.dy2 + (k21 * st.dx2 + k11 * st.dx1) * st.dy1;
        const T r = sampled - target[o1 + p.i];
        if (abar) {
            const T ddx = (k11 - k21) * st.dy1 + (k12 - k22) * st.dy2;
            const T ddy = (k11 * st.dx1 + k21 * st.dx2) - (k12 * st.dx1 + k22 * st.dx2);
            abar[2 * o1 + p.i] = r * ddx;
            abar[2 * o1 + P + p.i] = r * ddy;
        }
        contrib = r * r;
    }
    block_sum(contrib, partial);
}

// pbar += adjoint of C = phi_i o phi_i at every x (pbar zeroed by the caller).
//
// What bounds this is the float64 additions to global memory, ten per point.  Where the next
// lane's stencil continues this one's -- everywhere but at seams and strong stretches -- the
// right-hand samples' terms are handed to it and added to its left-hand ones, and the term of
// the point itself joins the sample that is the point: four additions per point (32 float64 grids of
// 256 x 128: 29.6 -> 22.2 us).
template <typename T>
__global__ void k_data_compose_adjoint(const T* __restrict__ f, const T* __restrict__ abar, T* __restrict__ pbar,
                                       int nx, int ny) {
    csg::pdl_begin();
    Pt p;
    const bool in = point(nx, ny, p);
    const int P = nx * ny;
    const size_t o2 = static_cast<size_t>(blockIdx.y) * 2 * P;
    const T* F = f + o2;
    T* out = pbar + o2;
    int at[4] = {-1, -1, -1, -1};  // 22, 12, 21, 11
    T term[2][4] = {};
    if (in) {
        const Stencil<T> st(F[p.i] - T(1), F[P + p.i] - T(1), nx, ny);
        at[0] = st.i22;
        at[1] = st.i12;
        at[2] = st.i21;
        at[3] = st.i11;
        T pos[2] = {T(0), T(0)};
        const Samples<T> f4(st, F, P);
        const T adjoint[2] = {abar[o2 + p.i], abar[o2 + P + p.i]};
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            const T period = static_cast<T>(ch == 0 ? nx : ny);
            const T c22 = f4.v[ch][0] - T(1);
            const T c12 = unwrap(f4.v[ch][1] - T(1), c22, period);
            const T c21 = unwrap(f4.v[ch][2] - T(1), c22, period);
            const T c11 = unwrap(f4.v[ch][3] - T(1), c22, period);
            const T a = adjoint[ch];
            pos[0] = pos[0] + a * ((c12 - c22) * st.dy2 + (c11 - c21) * st.dy1);
            pos[1] = pos[1] + a * ((c21 * st.dx2 + c11 * st.dx1) - (c22 * st.dx2 + c12 * st.dx1));
            term[ch][0] = a * (st.dx2 * st.dy2);
            term[ch][1] = a * (st.dx1 * st.dy2);
            term[ch][2] = a * (st.dx2 * st.dy1);
            term[ch][3] = a * (st.dx1 * st.dy1);
        }
        bool apart = true;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (apart && at[k] == p.i) {
                term[0][k] = term[0][k] + pos[0];
                term[1][k] = term[1][k] + pos[1];
                apart = false;
            }
        if (apart) {
            atomicAdd(out + p.i, pos[0]);
            atomicAdd(out + P + p.i, pos[1]);
        }
    }
    const int lane = threadIdx.x & 31;
    const int next_upper = __shfl_down_sync(0xffffffffu, at[0], 1), next_lower = __shfl_down_sync(0xffffffffu, at[2], 1);
    const bool give = in && lane < 31 && next_upper == at[1] && next_lower == at[3];
    const int given = __shfl_up_sync(0xffffffffu, static_cast<int>(give), 1);
    const bool take = given != 0 && lane > 0;
#pragma unroll
    for (int ch = 0; ch < 2; ++ch) {
        const T upper = __shfl_up_sync(0xffffffffu, term[ch][1], 1), lower = __shfl_up_sync(0xffffffffu, term[ch][3], 1);
        if (take) {
            term[ch][0] = term[ch][0] + upper;
            term[ch][2] = term[ch][2] + lower;
        }
        if (in) {
            T* o = out + ch * P;
            atomicAdd(o + at[0], term[ch][0]);
            atomicAdd(o + at[2], term[ch][2]);
            if (!give) {
                atomicAdd(o + at[1], term[ch][1]);
                atomicAdd(o + at[3], term[ch][3]);
            }
        }
    }
}

// grad = scale_b * s * abar (phi_0 = id + s v).
template <typename T>
__global__ void k_data_velocity_grad(const T* __restrict__ abar, const T* __restrict__ grad_scale, T s,
                                     T* __restrict__ grad, int nx, int ny) {
    csg::pdl_begin();
    Pt p;
    if (!point(nx, ny, p)) return;
    const int P = nx * ny;
    const size_t o2 = static_cast<size_t>(p.b) * 2 * P;
    const T g = grad_scale ? grad_scale[p.b] * s : s;
    grad[o2 + p.i] = abar[o2 + p.i] * g;
    grad[o2 + P + p.i] = abar[o2 + P + p.i] * g;
}

inline int data_checkpoints(int k, int every) { return k == 0 ? 1 : (k - 1) / every + 1; }

inline size_t align_up(size_t bytes) { return (bytes + 255) & ~static_cast<size_t>(255); }

template <typename T>
size_t data_scratch(int batch, int nx, int ny, int k, int every) {
    const size_t field = align_up(sizeof(T) * 2ULL * batch * nx * ny);
    const size_t nblocks = (static_cast<size_t>(nx) * ny + kThreads - 1) / kThreads;
    // forward ping-pong 2, backward segment `every`, abar + pbar, block partials
    return field * (2 + static_cast<size_t>(every) + 2) + align_up(sizeof(T) * nblocks * batch) + 256;
}

template <typename T>
struct DataScratch {
    T* work[2];
    T* seg;  // `every` maps
    T* abar;
    T* pbar;
    T* partial;
    size_t field_elems;
};

template <typename T>
DataScratch<T> carve_data(void* scratch, int batch, int nx, int ny, int every) {
    DataScratch<T> d{};
    const size_t field = align_up(sizeof(T) * 2ULL * batch * nx * ny);
    char* base = static_cast<char*>(scratch);
    d.work[0] = reinterpret_cast<T*>(base);
    d.work[1] = reinterpret_cast<T*>(base + field);
    d.seg = reinterpret_cast<T*>(base + 2 * field);
    d.abar = reinterpret_cast<T*>(base + (2 + static_cast<size_t>(every)) * field);
    d.pbar = reinterpret_cast<T*>(base + (3 + static_cast<size_t>(every)) * field);
    d.partial = reinterpret_cast<T*>(base + (4 + static_cast<size_t>(every)) * field);
    d.field_elems = field / sizeof(T);
    return d;
}

template <typename T>
int data_forward_typed(int batch, int nx, int ny, const T* v, const T* source, const T* target, int k, int every,
                       T* checkpoints, T* objective, void* scratch, size_t bytes, cudaStream_t s) {
    if (bytes < data_scratch<T>(batch, nx, ny, k, every)) return csg::fail(CSG_ERR_ARG, "data term: scratch too small");
    DataScratch<T> d = carve_data<T>(scratch, batch, nx, ny, every);
    const size_t field = 2ULL * batch * nx * ny;
    const dim3 g = grid_for(nx * ny, batch);
    const T step = static_cast<T>(std::ldexp(1.0, -k));
    (csg::note_launch(), csg::launch_pdl(k_smalldef<T>, g, kThreads, 0, s, v, checkpoints, nullptr, nx, ny, step, T(0)));
    const T* cur = checkpoints;
    for (int i = 1; i <= k; ++i) {
        T* dst = (i % every == 0 && i < k) ? checkpoints + field * (i / every) : d.work[i % 2];
        (csg::note_launch(), csg::launch_pdl(k_compose<T>, g, kThreads, 0, s, cur, nullptr, cur, nullptr, dst, nullptr, nx, ny));
        cur = dst;
    }
    (csg::note_launch(), csg::launch_pdl(k_data_sample<T>, g, kThreads, 0, s, source, target, cur, nullptr, d.partial, nx, ny));
    (csg::note_launch(), csg::launch_pdl(k_objective_out<T>, batch, csg::kOrderedThreads, 0, s, d.partial, static_cast<int>(g.x),
                                         objective));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

template <typename T>
int data_backward_typed(int batch, int nx, int ny, const T* source, const T* target, int k, int every,
                        const T* checkpoints, const T* grad_scale, T* grad, void* scratch, size_t bytes,
                        cudaStream_t s) {
    if (bytes < data_scratch<T>(batch, nx, ny, k, every)) return csg::fail(CSG_ERR_ARG, "data term: scratch too small");
    DataScratch<T> d = carve_data<T>(scratch, batch, nx, ny, every);
    const size_t field = 2ULL * batch * nx * ny;
    const dim3 g = grid_for(nx * ny, batch);
    const int n_ckpt = data_checkpoints(k, every);
    T* abar = d.abar;
    T* pbar = d.pbar;
    std::vector<const T*> maps(static_cast<size_t>(every) + 1);
    for (int j = n_ckpt - 1; j >= 0; --j) {
        const int first = j * every;
        const int last = (j == n_ckpt - 1) ? k : (j + 1) * every - 1;  // maps this segment needs
        maps[0] = checkpoints + field * j;
        for (int i = first + 1; i <= last; ++i) {
            T* dst = d.seg + d.field_elems * static_cast<size_t>(i - first - 1);
            (csg::note_launch(), csg::launch_pdl(k_compose<T>, g, kThreads, 0, s, maps[i - first - 1], nullptr, maps[i - first - 1],
                                                                   nullptr, dst, nullptr, nx, ny));
            maps[i - first] = dst;
        }
        if (j == n_ckpt - 1)
            (csg::note_launch(), csg::launch_pdl(k_data_sample<T>, g, kThreads, 0, s, source, target, maps[k - first], abar,
                                                                       d.partial, nx, ny));
        const int top = (j == n_ckpt - 1) ? k - 1 : last;
        for (int i = top; i >= first; --i) {
            CSG_CUDA_CHECK(cudaMemsetAsync(pbar, 0, sizeof(T) * field, s));
            (csg::note_launch(), csg::launch_pdl(k_data_compose_adjoint<T>, g, kThreads, 0, s, maps[i - first], abar, pbar, nx, ny));
            T* t = abar;
            abar = pbar;
            pbar = t;
        }
    }
    const T step = static_cast<T>(std::ldexp(1.0, -k));
    (csg::note_launch(), csg::launch_pdl(k_data_velocity_grad<T>, g, kThreads, 0, s, abar, grad_scale, step, grad, nx, ny));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int check_levels(int nx, int ny) {
    for (const auto& spec : grid_levels(nx, ny))
        if (!relax_supported(spec.first))
            return csg::fail(CSG_ERR_UNSUPPORTED,
                             "dartel: red-black relaxation needs an even x size on every multigrid level "
                             "(level %d x %d)", spec.second, spec.first);
    return CSG_OK;
}

}  // namespace

extern "C" {

size_t csg_dartel_scratch_bytes(int dtype, int batch, int nx, int ny) {
    if (!check_dtype(dtype) || batch < 1 || nx < 1 || ny < 1) return 0;
    return dtype == CSG_DTYPE_F64 ? step_bytes<double>(batch, nx, ny) : step_bytes<float>(batch, nx, ny);
}

int csg_dartel_solve(int dtype, int batch, int nx, int ny, const void* source_maps, const void* target_maps,
                     void* velocity, void* metrics, int loop, const double* params, int its, double lmreg, int cycles,
                     int nit, int code, int assume_initial_nonzero, void* scratch, size_t scratch_bytes,
                     csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!source_maps || !target_maps || !velocity || !metrics || !params || !scratch)
        return csg::fail(CSG_ERR_ARG, "dartel solve: null pointer");
    if (loop < 1 || its < 0 || cycles < 0 || nit < 0 || (code != 0 && code != 1) || loop > 30)
        return csg::fail(CSG_ERR_ARG, "dartel solve: bad loop/its/cycles/nit/code");
    rc = check_levels(nx, ny);
    if (rc) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == CSG_DTYPE_F64)
        return solve_typed<double>(source_maps, target_maps, velocity, metrics, batch, nx, ny, loop, params, its, lmreg,
                                   cycles, nit, code, assume_initial_nonzero, scratch, scratch_bytes, s);
    return solve_typed<float>(source_maps, target_maps, velocity, metrics, batch, nx, ny, loop, params, its, lmreg,
                              cycles, nit, code, assume_initial_nonzero, scratch, scratch_bytes, s);
}

int csg_dartel_step(int dtype, int batch, int nx, int ny, const void* source, const void* target, void* velocity,
                    void* metrics, int k, const double* params, double lmreg, int cycles, int nit, int code,
                    int assume_initial_nonzero, void* scratch, size_t scratch_bytes, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!source || !target || !velocity || !metrics || !params || !scratch)
        return csg::fail(CSG_ERR_ARG, "dartel step: null pointer");
    if (k < 0 || k > 30 || cycles < 0 || nit < 0 || (code != 0 && code != 1))
        return csg::fail(CSG_ERR_ARG, "dartel step: bad k/cycles/nit/code");
    rc = check_levels(nx, ny);
    if (rc) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == CSG_DTYPE_F64) {
        Arena ar{static_cast<char*>(scratch), scratch_bytes};
        StepBuffers<double> W;
        if (!W.carve(ar, batch, nx, ny)) return csg::fail(CSG_ERR_ARG, "dartel step: scratch too small");
        return dartel_step_impl<double>(W, static_cast<const double*>(source), static_cast<const double*>(target),
                                        static_cast<double*>(velocity), static_cast<double*>(metrics), 3, batch, nx, ny,
                                        k, params, lmreg, cycles, nit, code, assume_initial_nonzero, true, s);
    }
    Arena ar{static_cast<char*>(scratch), scratch_bytes};
    StepBuffers<float> W;
    if (!W.carve(ar, batch, nx, ny)) return csg::fail(CSG_ERR_ARG, "dartel step: scratch too small");
    return dartel_step_impl<float>(W, static_cast<const float*>(source), static_cast<const float*>(target),
                                   static_cast<float*>(velocity), static_cast<float*>(metrics), 3, batch, nx, ny, k,
                                   params, lmreg, cycles, nit, code, assume_initial_nonzero, true, s);
}

}  // extern "C"

// ------------------------------------------------------- single operators

namespace {

template <typename T>
int smalldef_typed(int batch, int nx, int ny, const void* v, double scale, void* map, void* jac, cudaStream_t s) {
    (csg::note_launch(), csg::launch_pdl(k_smalldef<T>, grid_for(nx * ny, batch), kThreads, 0, s, static_cast<const T*>(v), static_cast<T*>(map),
                                                                 static_cast<T*>(jac), nx, ny, T(scale), T(scale * 0.5)));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

template <typename T>
int squaring_typed(int batch, int nx, int ny, const void* rhs, const void* hess, const void* map, const void* jac,
                   int k, int save, void* b_out, void* a_out, void* map_out, void* jac_out, void* scratch_out,
                   void* work, size_t bytes, cudaStream_t s) {
    const size_t P = static_cast<size_t>(nx) * ny * batch;
    Arena ar{static_cast<char*>(work), bytes};
    T *rb[2], *ha[2], *maps[2], *jacs[2];
    for (int i = 0; i < 2; ++i) {
        rb[i] = ar.take<T>(2 * P);
        ha[i] = ar.take<T>(3 * P);
        maps[i] = ar.take<T>(2 * P);
        jacs[i] = ar.take<T>(4 * P);
    }
    if (!ar.ok) return csg::fail(CSG_ERR_ARG, "squaring: scratch too small");
    CSG_CUDA_CHECK(cudaMemcpyAsync(rb[0], rhs, 2 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    CSG_CUDA_CHECK(cudaMemcpyAsync(ha[0], hess, 3 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    CSG_CUDA_CHECK(cudaMemcpyAsync(maps[0], map, 2 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    CSG_CUDA_CHECK(cudaMemcpyAsync(jacs[0], jac, 4 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    Squaring<T> r = run_squaring<T>(rb, ha, maps, jacs, k, save != 0, batch, nx, ny, s);
    CSG_CUDA_CHECK(cudaMemcpyAsync(b_out, rb[r.cur_ba], 2 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    CSG_CUDA_CHECK(cudaMemcpyAsync(a_out, ha[r.cur_ba], 3 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    if (map_out) CSG_CUDA_CHECK(cudaMemcpyAsync(map_out, maps[r.cur_map], 2 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    if (jac_out) CSG_CUDA_CHECK(cudaMemcpyAsync(jac_out, jacs[r.cur_map], 4 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    if (scratch_out) CSG_CUDA_CHECK(cudaMemcpyAsync(scratch_out, maps[0], 2 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

template <typename T>
int expdef_typed(int batch, int nx, int ny, const void* v, int k, void* map_out, void* jac_out, void* work, size_t bytes,
                 cudaStream_t s) {
    const size_t P = static_cast<size_t>(nx) * ny * batch;
    Arena ar{static_cast<char*>(work), bytes};
    T* maps[2] = {ar.take<T>(2 * P), ar.take<T>(2 * P)};
    T* jacs[2] = {ar.take<T>(4 * P), ar.take<T>(4 * P)};
    if (!ar.ok) return csg::fail(CSG_ERR_ARG, "expdef: scratch too small");
    const double scale = 1.0 / static_cast<double>(1LL << k);
    const dim3 g = grid_for(nx * ny, batch);
    const bool with_jac = jac_out != nullptr;
    (csg::note_launch(), csg::launch_pdl(k_smalldef<T>, g, kThreads, 0, s, static_cast<const T*>(v), maps[0], with_jac ? jacs[0] : nullptr, nx, ny,
                                         T(scale), T(scale * 0.5)));
    int cur = 0;
    for (int i = 0; i < k; ++i) {
        (csg::note_launch(), csg::launch_pdl(k_compose<T>, g, kThreads, 0, s, maps[cur], with_jac ? jacs[cur] : nullptr, maps[cur],
                                            with_jac ? jacs[cur] : nullptr, maps[1 - cur],
                                            with_jac ? jacs[1 - cur] : nullptr, nx, ny));
        cur = 1 - cur;
    }
    CSG_CUDA_CHECK(cudaMemcpyAsync(map_out, maps[cur], 2 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    if (with_jac) CSG_CUDA_CHECK(cudaMemcpyAsync(jac_out, jacs[cur], 4 * P * sizeof(T), cudaMemcpyDeviceToDevice, s));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

template <typename T>
int fmg_typed(int batch, int nx, int ny, const void* hess, const void* rhs, const double* params, int cycles, int nit,
              void* u, int has_initial, int assume_nonzero, void* work, size_t bytes, cudaStream_t s,
              double timeout_s = 2.0, int silent = -1) {
    const size_t P = static_cast<size_t>(nx) * ny * batch;
    Arena ar{static_cast<char*>(work), bytes};
    FmgBuffers<T> buf;
    buf.take_control(ar);
    if (!buf.carve(ar, batch, nx, ny)) return csg::fail(CSG_ERR_ARG, "fmg: scratch too small");
    CSG_CUDA_CHECK(cudaMemsetAsync(buf.ctl, 0, sizeof(csg::Control), s));
    buf.A[0] = const_cast<T*>(static_cast<const T*>(hess));
    buf.B[0] = const_cast<T*>(static_cast<const T*>(rhs));
    buf.U[0] = static_cast<T*>(u);
    bool coarse_init = !has_initial;
    if (has_initial && !assume_nonzero) {
        int flag = 0;
        (csg::note_launch(), csg::launch_pdl(k_any_nonzero<T>, static_cast<unsigned>((2 * P + kThreads - 1) / kThreads), kThreads, 0, s, buf.U[0], 2 * P,
                                                                                                     buf.flag));
        CSG_CUDA_CHECK(cudaMemcpyAsync(&flag, buf.flag, sizeof(int), cudaMemcpyDeviceToHost, s));
        CSG_CUDA_CHECK(cudaStreamSynchronize(s));
        coarse_init = flag == 0;
    }
    if (coarse_init) CSG_CUDA_CHECK(cudaMemsetAsync(u, 0, 2 * P * sizeof(T), s));
    Fmg<T> fmg{buf, batch, {params[0], params[1], params[2], params[3], params[4]}, cycles, nit, s, nx, ny, timeout_s, silent};
    fmg.run(coarse_init);
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

}  // namespace

extern "C" {

int csg_dartel_smalldef(int dtype, int batch, int nx, int ny, const void* velocity, double scale, void* map_out,
                        void* jac_out, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!velocity || (!map_out && !jac_out)) return csg::fail(CSG_ERR_ARG, "smalldef: null pointer");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    return dtype == CSG_DTYPE_F64 ? smalldef_typed<double>(batch, nx, ny, velocity, scale, map_out, jac_out, s)
                                  : smalldef_typed<float>(batch, nx, ny, velocity, scale, map_out, jac_out, s);
}

int csg_dartel_compose(int dtype, int batch, int nx, int ny, const void* a, const void* ja, const void* b,
                       const void* jb, void* c_out, void* jc_out, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!a || !b || !c_out || ((ja != nullptr) != (jb != nullptr)) || ((ja != nullptr) != (jc_out != nullptr)))
        return csg::fail(CSG_ERR_ARG, "compose: null pointer or partial Jacobian set");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const dim3 g = grid_for(nx * ny, batch);
    if (dtype == CSG_DTYPE_F64)
        (csg::note_launch(), csg::launch_pdl(k_compose<double>, g, kThreads, 0, s, static_cast<const double*>(a), static_cast<const double*>(ja),
                                                 static_cast<const double*>(b), static_cast<const double*>(jb),
                                                 static_cast<double*>(c_out), static_cast<double*>(jc_out), nx, ny));
    else
        (csg::note_launch(), csg::launch_pdl(k_compose<float>, g, kThreads, 0, s, static_cast<const float*>(a), static_cast<const float*>(ja),
                                                static_cast<const float*>(b), static_cast<const float*>(jb),
                                                static_cast<float*>(c_out), static_cast<float*>(jc_out), nx, ny));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_dartel_jac_div(int dtype, int batch, int nx, int ny, const void* jac, const void* velocity, double scale,
                       void* out, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!jac || !velocity || !out) return csg::fail(CSG_ERR_ARG, "jac_div: null pointer");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const dim3 g = grid_for(nx * ny, batch);
    if (dtype == CSG_DTYPE_F64)
        (csg::note_launch(), csg::launch_pdl(k_jacdiv<double>, g, kThreads, 0, s, static_cast<const double*>(jac), static_cast<const double*>(velocity),
                                                static_cast<double*>(out), nx, ny, scale * 0.5));
    else
        (csg::note_launch(), csg::launch_pdl(k_jacdiv<float>, g, kThreads, 0, s, static_cast<const float*>(jac), static_cast<const float*>(velocity),
                                               static_cast<float*>(out), nx, ny, static_cast<float>(scale * 0.5)));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_dartel_objfun(int dtype, int batch, int nx, int ny, const void* source, const void* target, const void* map,
                      const void* jac, const void* weights, void* rhs_out, void* hess_out, void* objective_out,
                      void* scratch, size_t scratch_bytes, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!source || !target || !map || !jac || !rhs_out || !hess_out || !objective_out || !scratch)
        return csg::fail(CSG_ERR_ARG, "objfun: null pointer");
    const int nblocks = (nx * ny + kThreads - 1) / kThreads;
    if (scratch_bytes < static_cast<size_t>(nblocks) * batch * dtype_size(dtype))
        return csg::fail(CSG_ERR_ARG, "objfun: scratch too small");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const dim3 g = grid_for(nx * ny, batch);
    if (dtype == CSG_DTYPE_F64) {
        (csg::note_launch(), csg::launch_pdl(k_objfun<double, false>, g, kThreads, 0, s, 
            static_cast<const double*>(source), static_cast<const double*>(target), static_cast<const double*>(map),
            static_cast<const double*>(jac), nullptr, static_cast<const double*>(weights), static_cast<double*>(rhs_out),
            static_cast<double*>(hess_out), static_cast<double*>(scratch), nx, ny, 0.0));
        (csg::note_launch(), csg::launch_pdl(k_objective_out<double>, batch, csg::kOrderedThreads, 0, s, static_cast<double*>(scratch), nblocks,
                                                     static_cast<double*>(objective_out)));
    } else {
        (csg::note_launch(), csg::launch_pdl(k_objfun<float, false>, g, kThreads, 0, s, 
            static_cast<const float*>(source), static_cast<const float*>(target), static_cast<const float*>(map),
            static_cast<const float*>(jac), nullptr, static_cast<const float*>(weights), static_cast<float*>(rhs_out),
            static_cast<float*>(hess_out), static_cast<float*>(scratch), nx, ny, 0.0f));
        (csg::note_launch(), csg::launch_pdl(k_objective_out<float>, batch, csg::kOrderedThreads, 0, s, static_cast<float*>(scratch), nblocks,
                                                    static_cast<float*>(objective_out)));
    }
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_dartel_squaring(int dtype, int batch, int nx, int ny, const void* rhs, const void* hess, const void* map,
                        const void* jac, int k, int save_transformation, void* b_out, void* a_out, void* map_out,
                        void* jac_out, void* scratch_map_out, void* scratch, size_t scratch_bytes,
                        csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!rhs || !hess || !map || !jac || !b_out || !a_out || !scratch || k < 0 || k > 30)
        return csg::fail(CSG_ERR_ARG, "squaring: null pointer or bad k");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == CSG_DTYPE_F64)
        return squaring_typed<double>(batch, nx, ny, rhs, hess, map, jac, k, save_transformation, b_out, a_out, map_out,
                                      jac_out, scratch_map_out, scratch, scratch_bytes, s);
    return squaring_typed<float>(batch, nx, ny, rhs, hess, map, jac, k, save_transformation, b_out, a_out, map_out,
                                 jac_out, scratch_map_out, scratch, scratch_bytes, s);
}

int csg_dartel_regularization(int dtype, int batch, int nx, int ny, const void* velocity, const double* params,
                              int rtype, void* out, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!velocity || !params || !out || rtype < 0 || rtype > 2)
        return csg::fail(CSG_ERR_ARG, "regularization: null pointer or rtype not in {0, 1, 2}");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const RegWeights rw = reg_weights(params, rtype);
    const dim3 g = grid_for(nx * ny, batch);
    if (dtype == CSG_DTYPE_F64)
        (csg::note_launch(), csg::launch_pdl(k_regularise<double>, g, kThreads, 0, s, static_cast<const double*>(velocity), static_cast<double*>(out), nx,
                                                    ny, rtype, rw));
    else
        (csg::note_launch(), csg::launch_pdl(k_regularise<float>, g, kThreads, 0, s, static_cast<const float*>(velocity), static_cast<float*>(out), nx, ny,
                                                   rtype, rw));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_dartel_membrane_apply(int dtype, int batch, int nx, int ny, const void* hess, const void* field,
                              const double* params, void* out, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!hess || !field || !params || !out) return csg::fail(CSG_ERR_ARG, "membrane apply: null pointer");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const RegWeights rw = reg_weights(params, 1);
    const dim3 g = grid_for(nx * ny, batch);
    if (dtype == CSG_DTYPE_F64)
        (csg::note_launch(), csg::launch_pdl(k_membrane_apply<double>, g, kThreads, 0, s, static_cast<const double*>(hess), static_cast<const double*>(field),
                                                        nullptr, static_cast<double*>(out), nx, ny, rw));
    else
        (csg::note_launch(), csg::launch_pdl(k_membrane_apply<float>, g, kThreads, 0, s, static_cast<const float*>(hess), static_cast<const float*>(field),
                                                       nullptr, static_cast<float*>(out), nx, ny, rw));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_dartel_relax(int dtype, int batch, int nx, int ny, const void* hess, const void* rhs, const double* params,
                     int nit, void* u, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!hess || !rhs || !params || !u || nit < 0) return csg::fail(CSG_ERR_ARG, "relax: null pointer or nit < 0");
    if (!relax_supported(nx))
        return csg::fail(CSG_ERR_UNSUPPORTED, "relax: red-black relaxation on the GPU needs an even x size (got %d)", nx);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const MemWeights w = mem_weights(params);
    const dim3 g = grid_for(nx * ny, batch);
    for (int it = 0; it < 2 * nit; ++it) {
        const int colour = it % 2 == 0 ? 1 : 0;
        if (dtype == CSG_DTYPE_F64)
            (csg::note_launch(), csg::launch_pdl(k_relax<double>, g, kThreads, 0, s, static_cast<const double*>(hess), static_cast<const double*>(rhs),
                                                   static_cast<double*>(u), nx, ny, colour, w.w00, w.w01, w.w10));
        else
            (csg::note_launch(), csg::launch_pdl(k_relax<float>, g, kThreads, 0, s, static_cast<const float*>(hess), static_cast<const float*>(rhs),
                                                  static_cast<float*>(u), nx, ny, colour, static_cast<float>(w.w00),
                                                  static_cast<float>(w.w01), static_cast<float>(w.w10)));
    }
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_dartel_resize(int dtype, int fields, int src_nx, int src_ny, const void* src, int dst_nx, int dst_ny,
                      void* dst, int accumulate, csg_stream_t stream) {
    if (!check_dtype(dtype) || fields < 1 || src_nx < 1 || src_ny < 1 || dst_nx < 1 || dst_ny < 1 || !src || !dst)
        return csg::fail(CSG_ERR_ARG, "resize: bad arguments");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const dim3 g = grid_for(dst_nx * dst_ny, fields);
    if (dtype == CSG_DTYPE_F64)
        (csg::note_launch(), csg::launch_pdl(k_resize<double>, g, kThreads, 0, s, static_cast<const double*>(src), static_cast<double*>(dst), src_nx,
                                                src_ny, dst_nx, dst_ny, accumulate));
    else
        (csg::note_launch(), csg::launch_pdl(k_resize<float>, g, kThreads, 0, s, static_cast<const float*>(src), static_cast<float*>(dst), src_nx, src_ny,
                                               dst_nx, dst_ny, accumulate));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_dartel_fmg(int dtype, int batch, int nx, int ny, const void* hess, const void* rhs, const double* params,
                   int cycles, int nit, void* u, int has_initial, int assume_initial_nonzero, void* scratch,
                   size_t scratch_bytes, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!hess || !rhs || !params || !u || !scratch || cycles < 0 || nit < 0)
        return csg::fail(CSG_ERR_ARG, "fmg: null pointer or negative cycles / nit");
    rc = check_levels(nx, ny);
    if (rc) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == CSG_DTYPE_F64)
        return fmg_typed<double>(batch, nx, ny, hess, rhs, params, cycles, nit, u, has_initial, assume_initial_nonzero,
                                 scratch, scratch_bytes, s);
    return fmg_typed<float>(batch, nx, ny, hess, rhs, params, cycles, nit, u, has_initial, assume_initial_nonzero,
                            scratch, scratch_bytes, s);
}

int csg_selftest_exchange_timeout(int dtype, int batch, int nx, int ny, const void* hess, const void* rhs,
                                  const double* params, int cycles, int nit, void* u, void* scratch,
                                  size_t scratch_bytes, double timeout_s, int silent, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!hess || !rhs || !params || !u || !scratch || cycles < 0 || nit < 0 || !(timeout_s > 0.0) || timeout_s > 10.0)
        return csg::fail(CSG_ERR_ARG, "exchange self-test: null pointer, negative cycles / nit or no 0 < timeout_s <= 10");
    rc = check_levels(nx, ny);
    if (rc) return rc;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    return dtype == CSG_DTYPE_F64
               ? fmg_typed<double>(batch, nx, ny, hess, rhs, params, cycles, nit, u, 1, 1, scratch, scratch_bytes, s, timeout_s, silent)
               : fmg_typed<float>(batch, nx, ny, hess, rhs, params, cycles, nit, u, 1, 1, scratch, scratch_bytes, s, timeout_s, silent);
}

int csg_dartel_expdef(int dtype, int batch, int nx, int ny, const void* velocity, int k, void* map_out, void* jac_out,
                      void* scratch, size_t scratch_bytes, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!velocity || !map_out || !scratch || k < 0 || k > 30)
        return csg::fail(CSG_ERR_ARG, "expdef: null pointer or bad k");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == CSG_DTYPE_F64)
        return expdef_typed<double>(batch, nx, ny, velocity, k, map_out, jac_out, scratch, scratch_bytes, s);
    return expdef_typed<float>(batch, nx, ny, velocity, k, map_out, jac_out, scratch, scratch_bytes, s);
}

size_t csg_dartel_data_scratch_bytes(int dtype, int batch, int nx, int ny, int k, int checkpoint_every) {
    if (!check_dtype(dtype) || batch < 1 || nx < 1 || ny < 1 || k < 0 || k > 30 || checkpoint_every < 1) return 0;
    return dtype == CSG_DTYPE_F64 ? data_scratch<double>(batch, nx, ny, k, checkpoint_every)
                                  : data_scratch<float>(batch, nx, ny, k, checkpoint_every);
}

int csg_dartel_data_checkpoints(int k, int checkpoint_every) {
    if (k < 0 || k > 30 || checkpoint_every < 1) return 0;
    return data_checkpoints(k, checkpoint_every);
}

int csg_dartel_data_forward(int dtype, int batch, int nx, int ny, const void* velocity, const void* source,
                            const void* target, int k, int checkpoint_every, void* checkpoints, void* objective,
                            void* scratch, size_t scratch_bytes, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!velocity || !source || !target || !checkpoints || !objective || !scratch || k < 0 || k > 30 ||
        checkpoint_every < 1)
        return csg::fail(CSG_ERR_ARG, "data term forward: null pointer, bad k or checkpoint interval");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == CSG_DTYPE_F64)
        return data_forward_typed<double>(batch, nx, ny, static_cast<const double*>(velocity),
                                          static_cast<const double*>(source), static_cast<const double*>(target), k,
                                          checkpoint_every, static_cast<double*>(checkpoints),
                                          static_cast<double*>(objective), scratch, scratch_bytes, s);
    return data_forward_typed<float>(batch, nx, ny, static_cast<const float*>(velocity),
                                     static_cast<const float*>(source), static_cast<const float*>(target), k,
                                     checkpoint_every, static_cast<float*>(checkpoints), static_cast<float*>(objective),
                                     scratch, scratch_bytes, s);
}

int csg_dartel_data_backward(int dtype, int batch, int nx, int ny, const void* source, const void* target, int k,
                             int checkpoint_every, const void* checkpoints, const void* grad_scale,
                             void* grad_velocity, void* scratch, size_t scratch_bytes, csg_stream_t stream) {
    int rc = check_grid(dtype, batch, nx, ny);
    if (rc) return rc;
    if (!source || !target || !checkpoints || !grad_velocity || !scratch || k < 0 || k > 30 || checkpoint_every < 1)
        return csg::fail(CSG_ERR_ARG, "data term backward: null pointer, bad k or checkpoint interval");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (dtype == CSG_DTYPE_F64)
        return data_backward_typed<double>(batch, nx, ny, static_cast<const double*>(source),
                                           static_cast<const double*>(target), k, checkpoint_every,
                                           static_cast<const double*>(checkpoints),
                                           static_cast<const double*>(grad_scale), static_cast<double*>(grad_velocity),
                                           scratch, scratch_bytes, s);
    return data_backward_typed<float>(batch, nx, ny, static_cast<const float*>(source),
                                      static_cast<const float*>(target), k, checkpoint_every,
                                      static_cast<const float*>(checkpoints), static_cast<const float*>(grad_scale),
                                      static_cast<float*>(grad_velocity), scratch, scratch_bytes, s);
}

}  // extern "C"
