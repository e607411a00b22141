// Surf2Sphere ordered area-smoothing sweeps as ONE persistent cooperative
// kernel for sm_100a.
//
// Semantics follow the reference's ordered Gauss-Seidel sweeps
// (src/cat_surface_gpu/surf2sphere.py:35-280 and 1039-1092): every vertex,
// in index order, moves to the area-weighted centroid of its incident faces
// (faces in ascending id, areas clamped to [0, 1]); after sweep s with
// s % project_every == 0 all points are projected to `radius`.
//
// Schedule: instead of one launch per dependency level per sweep (the
// reference launches sum(levels) x 4,999 kernels), vertex v of sweep s runs at
// wavefront step s * stride + level(v) inside one launch.  With
// stride = 1 + max_{edges v<w} (level(w) - level(v)) every read sees exactly
// the value the sequential order would see (lower neighbours: this sweep;
// higher neighbours: previous sweep), so the in-place buffer needs no copy.
// Steps are separated by a bounded grid barrier; projections drain the
// wavefront (one barrier before and after).
//
// Data layout: positions live in a float4 (or double4) working copy in HBM
// (L2-resident for cortical meshes), read with 16-byte ld.global.cg loads so
// no stale L1 line can be observed across steps.  Each vertex's incident
// faces are stored CSR-contiguous as int4 {v0, v1, v2, face}: a group of G
// lanes reads G consecutive slots (coalesced), computes one face per lane and
// accumulates the per-face terms in slot order through warp shuffles, which
// keeps the reference's sequential accumulation order exactly.
//
// Arithmetic: CSG_ARITH_CAT reproduces the reference's mixed precision
// (float32 edge/cross/sum-of-squares, float64 sqrt/centre/accumulate/divide,
// float32 store) with one IEEE rounding per operation (explicit _rn
// intrinsics, no contraction), so results are bit-identical to the CPU
// restatement compiled with -ffp-contract=off.
#include <cstdint>
#include <mutex>

#include <cuda_runtime.h>

#include "common.cuh"
#include "cooperative.h"
#include "errors.h"

namespace {

constexpr unsigned kFull = 0xffffffffu;

struct ArealParams {
    void* points;  // caller's [n,3] float32 or float64
    void* work;    // float4[n] or double4[n] working copy (scratch)
    csg::Control* ctl;
    const int4* slot_tri;
    const int* slot_off;
    const int* order;
    const int* level_begin;
    const int* level_end;
    int n;
    int n_levels;
    int stride;
    int max_degree;
    int nloc_max;  // vertices owned by one CTA (set at launch)
    int iterations;
    int project_every;
    int allow_dataflow;  // float32 modes: published (position, version) words instead of per-step barriers
    unsigned int epoch_magic;  // ceil(2^32 / project_every), 0: divide (see epoch_rest)
    double radius;
    unsigned long long timeout_ns;
};

struct alignas(32) D4 {
    double x, y, z, w;
};

template <int MODE>
struct Traits;

// CAT mixed: float32 storage, float64 accumulation.
template <>
struct Traits<CSG_ARITH_CAT> {
    using Store = float4;
    using Acc = double;
    struct P3 {
        float x, y, z;
    };
    static __device__ __forceinline__ P3 load(const void* w, int v) {
        float4 q = __ldcg(static_cast<const float4*>(w) + v);
        return {q.x, q.y, q.z};
    }
    static __device__ __forceinline__ void face(const P3& a, const P3& b, const P3& c, double& area, double& mx,
                                                double& my, double& mz) {
        float e0x = __fsub_rn(b.x, a.x), e0y = __fsub_rn(b.y, a.y), e0z = __fsub_rn(b.z, a.z);
        float e1x = __fsub_rn(c.x, a.x), e1y = __fsub_rn(c.y, a.y), e1z = __fsub_rn(c.z, a.z);
        float cx = __fsub_rn(__fmul_rn(e0y, e1z), __fmul_rn(e0z, e1y));
        float cy = __fsub_rn(__fmul_rn(e0z, e1x), __fmul_rn(e0x, e1z));
        float cz = __fsub_rn(__fmul_rn(e0x, e1y), __fmul_rn(e0y, e1x));
        float sq = __fadd_rn(__fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy)), __fmul_rn(cz, cz));
        area = __dmul_rn(0.5, __dsqrt_rn(static_cast<double>(sq)));
        mx = csg::div3_rn(__dadd_rn(__dadd_rn((double)a.x, (double)b.x), (double)c.x));
        my = csg::div3_rn(__dadd_rn(__dadd_rn((double)a.y, (double)b.y), (double)c.y));
        mz = csg::div3_rn(__dadd_rn(__dadd_rn((double)a.z, (double)b.z), (double)c.z));
        area = area > 0.0 ? area : 0.0;
        area = area < 1.0 ? area : 1.0;
    }
    static __device__ __forceinline__ void store(void* w, int v, double total, double wx, double wy, double wz) {
        double safe = total > 1.0e-20 ? total : 1.0e-20;
        float4 q = make_float4(__double2float_rn(__ddiv_rn(wx, safe)), __double2float_rn(__ddiv_rn(wy, safe)),
                               __double2float_rn(__ddiv_rn(wz, safe)), 0.0f);
        __stcg(static_cast<float4*>(w) + v, q);
    }
    static __device__ __forceinline__ P3 project_p3(const P3& q, double radius) {
        float sq = __fadd_rn(__fadd_rn(__fmul_rn(q.x, q.x), __fmul_rn(q.y, q.y)), __fmul_rn(q.z, q.z));
        double norm = __dsqrt_rn(static_cast<double>(sq));
        double scale = __ddiv_rn(radius, norm > 1.0e-20 ? norm : 1.0e-20);
        return {__double2float_rn(__dmul_rn((double)q.x, scale)), __double2float_rn(__dmul_rn((double)q.y, scale)),
                __double2float_rn(__dmul_rn((double)q.z, scale))};
    }
    static __device__ __forceinline__ void project(void* w, int v, double radius) {
        const P3 q = project_p3(load(w, v), radius);
        __stcg(static_cast<float4*>(w) + v, make_float4(q.x, q.y, q.z, 0.0f));
    }
    static __device__ __forceinline__ void pack(const void* in, void* w, int v) {
        const float* p = static_cast<const float*>(in) + 3LL * v;
        static_cast<float4*>(w)[v] = make_float4(p[0], p[1], p[2], 0.0f);
    }
    static __device__ __forceinline__ void unpack(const void* w, void* out, int v) {
        float4 q = __ldcg(static_cast<const float4*>(w) + v);
        float* p = static_cast<float*>(out) + 3LL * v;
        p[0] = q.x;
        p[1] = q.y;
        p[2] = q.z;
    }
};

// Plain float32 storage and arithmetic.
template <>
struct Traits<CSG_ARITH_FP32> {
    using Acc = float;
    using P3 = Traits<CSG_ARITH_CAT>::P3;
    static __device__ __forceinline__ P3 load(const void* w, int v) { return Traits<CSG_ARITH_CAT>::load(w, v); }
    static __device__ __forceinline__ void face(const P3& a, const P3& b, const P3& c, float& area, float& mx,
                                                float& my, float& mz) {
        float e0x = __fsub_rn(b.x, a.x), e0y = __fsub_rn(b.y, a.y), e0z = __fsub_rn(b.z, a.z);
        float e1x = __fsub_rn(c.x, a.x), e1y = __fsub_rn(c.y, a.y), e1z = __fsub_rn(c.z, a.z);
        float cx = __fsub_rn(__fmul_rn(e0y, e1z), __fmul_rn(e0z, e1y));
        float cy = __fsub_rn(__fmul_rn(e0z, e1x), __fmul_rn(e0x, e1z));
        float cz = __fsub_rn(__fmul_rn(e0x, e1y), __fmul_rn(e0y, e1x));
        float sq = __fadd_rn(__fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy)), __fmul_rn(cz, cz));
        area = __fmul_rn(0.5f, __fsqrt_rn(sq));
        mx = __fdiv_rn(__fadd_rn(__fadd_rn(a.x, b.x), c.x), 3.0f);
        my = __fdiv_rn(__fadd_rn(__fadd_rn(a.y, b.y), c.y), 3.0f);
        mz = __fdiv_rn(__fadd_rn(__fadd_rn(a.z, b.z), c.z), 3.0f);
        area = area > 0.0f ? area : 0.0f;
        area = area < 1.0f ? area : 1.0f;
    }
    static __device__ __forceinline__ void store(void* w, int v, float total, float wx, float wy, float wz) {
        float safe = total > 1.0e-20f ? total : 1.0e-20f;
        __stcg(static_cast<float4*>(w) + v,
               make_float4(__fdiv_rn(wx, safe), __fdiv_rn(wy, safe), __fdiv_rn(wz, safe), 0.0f));
    }
    static __device__ __forceinline__ P3 project_p3(const P3& q, double radius) {
        const float r = static_cast<float>(radius);
        float sq = __fadd_rn(__fadd_rn(__fmul_rn(q.x, q.x), __fmul_rn(q.y, q.y)), __fmul_rn(q.z, q.z));
        float norm = __fsqrt_rn(sq);
        float scale = __fdiv_rn(r, norm > 1.0e-20f ? norm : 1.0e-20f);
        return {__fmul_rn(q.x, scale), __fmul_rn(q.y, scale), __fmul_rn(q.z, scale)};
    }
    static __device__ __forceinline__ void project(void* w, int v, double radius) {
        const P3 q = project_p3(load(w, v), radius);
        __stcg(static_cast<float4*>(w) + v, make_float4(q.x, q.y, q.z, 0.0f));
    }
    static __device__ __forceinline__ void pack(const void* in, void* w, int v) { Traits<CSG_ARITH_CAT>::pack(in, w, v); }
    static __device__ __forceinline__ void unpack(const void* w, void* out, int v) {
        Traits<CSG_ARITH_CAT>::unpack(w, out, v);
    }
};

// Float64 storage and arithmetic.
template <>
struct Traits<CSG_ARITH_FP64> {
    using Acc = double;
    struct P3 {
        double x, y, z;
    };
    static __device__ __forceinline__ P3 load(const void* w, int v) {
        const double2* base = reinterpret_cast<const double2*>(static_cast<const D4*>(w) + v);
        double2 xy = __ldcg(base);
        double2 zw = __ldcg(base + 1);
        return {xy.x, xy.y, zw.x};
    }
    static __device__ __forceinline__ void face(const P3& a, const P3& b, const P3& c, double& area, double& mx,
                                                double& my, double& mz) {
        double e0x = __dsub_rn(b.x, a.x), e0y = __dsub_rn(b.y, a.y), e0z = __dsub_rn(b.z, a.z);
        double e1x = __dsub_rn(c.x, a.x), e1y = __dsub_rn(c.y, a.y), e1z = __dsub_rn(c.z, a.z);
        double cx = __dsub_rn(__dmul_rn(e0y, e1z), __dmul_rn(e0z, e1y));
        double cy = __dsub_rn(__dmul_rn(e0z, e1x), __dmul_rn(e0x, e1z));
        double cz = __dsub_rn(__dmul_rn(e0x, e1y), __dmul_rn(e0y, e1x));
        double sq = __dadd_rn(__dadd_rn(__dmul_rn(cx, cx), __dmul_rn(cy, cy)), __dmul_rn(cz, cz));
        area = __dmul_rn(0.5, __dsqrt_rn(sq));
        mx = csg::div3_rn(__dadd_rn(__dadd_rn(a.x, b.x), c.x));
        my = csg::div3_rn(__dadd_rn(__dadd_rn(a.y, b.y), c.y));
        mz = csg::div3_rn(__dadd_rn(__dadd_rn(a.z, b.z), c.z));
        area = area > 0.0 ? area : 0.0;
        area = area < 1.0 ? area : 1.0;
    }
    static __device__ __forceinline__ void write(void* w, int v, double x, double y, double z) {
        double2* base = reinterpret_cast<double2*>(static_cast<D4*>(w) + v);
        __stcg(base, make_double2(x, y));
        __stcg(base + 1, make_double2(z, 0.0));
    }
    static __device__ __forceinline__ void store(void* w, int v, double total, double wx, double wy, double wz) {
        double safe = total > 1.0e-20 ? total : 1.0e-20;
        write(w, v, __ddiv_rn(wx, safe), __ddiv_rn(wy, safe), __ddiv_rn(wz, safe));
    }
    static __device__ __forceinline__ void project(void* w, int v, double radius) {
        P3 q = load(w, v);
        double sq = __dadd_rn(__dadd_rn(__dmul_rn(q.x, q.x), __dmul_rn(q.y, q.y)), __dmul_rn(q.z, q.z));
        double norm = __dsqrt_rn(sq);
        double scale = __ddiv_rn(radius, norm > 1.0e-20 ? norm : 1.0e-20);
        write(w, v, __dmul_rn(q.x, scale), __dmul_rn(q.y, scale), __dmul_rn(q.z, scale));
    }
    static __device__ __forceinline__ void pack(const void* in, void* w, int v) {
        const double* p = static_cast<const double*>(in) + 3LL * v;
        write(w, v, p[0], p[1], p[2]);
    }
    static __device__ __forceinline__ void unpack(const void* w, void* out, int v) {
        P3 q = load(w, v);
        double* p = static_cast<double*>(out) + 3LL * v;
        p[0] = q.x;
        p[1] = q.y;
        p[2] = q.z;
    }
};

template <typename T>
__device__ __forceinline__ T dadd(T a, T b);
template <>
__device__ __forceinline__ double dadd<double>(double a, double b) { return __dadd_rn(a, b); }
template <>
__device__ __forceinline__ float dadd<float>(float a, float b) { return __fadd_rn(a, b); }
template <typename T>
__device__ __forceinline__ T dmul(T a, T b);
template <>
__device__ __forceinline__ double dmul<double>(double a, double b) { return __dmul_rn(a, b); }
template <>
__device__ __forceinline__ float dmul<float>(float a, float b) { return __fmul_rn(a, b); }

// One vertex update by a group of G lanes.  All 32 lanes of the warp must
// call this together (warp shuffles); inactive groups pass v < 0.  `tri`
// points at the vertex's incident-face slots (shared or global memory).
//
// float64 accumulation (CAT and FP64 modes): every lane computes one face's
// area and area-weighted centre products and stages them in shared memory;
// lanes 0, 1 and 2 of the group then each sum, in slot order, the area
// total and one coordinate's weighted sum and divide it -- three dependent
// chains and three divides in parallel instead of one lane doing all four
// sums and three divides.  The arithmetic is unchanged: same products, same
// order of additions.
template <int MODE, int G, bool SMEM>
__device__ __forceinline__ void update_vertex(const ArealParams& p, int v, const int4* tri, int deg,
                                              double (*stage)[32]) {
    using T = Traits<MODE>;
    using Acc = typename T::Acc;
    const int lane = threadIdx.x & 31;
    const int glane = lane & (G - 1);
    const int gbase = lane & ~(G - 1);
    if (v < 0) deg = 0;
    const int wdeg = __reduce_max_sync(kFull, deg);
    if constexpr (sizeof(Acc) == 8) {
        double total = 0, wsum = 0;
        const double* mine = stage[1 + (glane < 3 ? glane : 0)];
        for (int c0 = 0; c0 < wdeg; c0 += G) {
            const int j = c0 + glane;
            double fa = 0, fx = 0, fy = 0, fz = 0;
            if (j < deg) {
                const int4 t = SMEM ? tri[j] : __ldg(tri + j);
                auto a = T::load(p.work, t.x);
                auto b = T::load(p.work, t.y);
                auto c = T::load(p.work, t.z);
                double mx, my, mz;
                T::face(a, b, c, fa, mx, my, mz);
                fx = __dmul_rn(fa, mx);
                fy = __dmul_rn(fa, my);
                fz = __dmul_rn(fa, mz);
            }
            stage[0][lane] = fa;
            stage[1][lane] = fx;
            stage[2][lane] = fy;
            stage[3][lane] = fz;
            __syncwarp();
            if (glane < 3) {
                const int n = min(G, deg - c0);
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    if (q < n) {  // slot order == ascending face id
                        total = __dadd_rn(total, stage[0][gbase + q]);
                        wsum = __dadd_rn(wsum, mine[gbase + q]);
                    }
                }
            }
            __syncwarp();
        }
        const bool write = v >= 0 && total > 0.0;
        const double safe = total > 1.0e-20 ? total : 1.0e-20;
        const double comp = (glane < 3 && write) ? __ddiv_rn(wsum, safe) : 0.0;
        if constexpr (MODE == CSG_ARITH_CAT) {
            const float cf = __double2float_rn(comp);
            const float cy = __shfl_sync(kFull, cf, gbase + 1);
            const float cz = __shfl_sync(kFull, cf, gbase + 2);
            if (write && glane == 0) __stcg(static_cast<float4*>(p.work) + v, make_float4(cf, cy, cz, 0.0f));
        } else {
            const double cy = __shfl_sync(kFull, comp, gbase + 1);
            const double cz = __shfl_sync(kFull, comp, gbase + 2);
            if (write && glane == 0) T::write(p.work, v, comp, cy, cz);
        }
    } else {
        Acc total = 0, wx = 0, wy = 0, wz = 0;
        for (int c0 = 0; c0 < wdeg; c0 += G) {
            const int j = c0 + glane;
            Acc fa = 0, fx = 0, fy = 0, fz = 0;
            if (j < deg) {
                const int4 t = SMEM ? tri[j] : __ldg(tri + j);
                auto a = T::load(p.work, t.x);
                auto b = T::load(p.work, t.y);
                auto c = T::load(p.work, t.z);
                T::face(a, b, c, fa, fx, fy, fz);
            }
#pragma unroll
            for (int q = 0; q < G; ++q) {
                const Acc a = __shfl_sync(kFull, fa, gbase + q);
                const Acc x = __shfl_sync(kFull, fx, gbase + q);
                const Acc y = __shfl_sync(kFull, fy, gbase + q);
                const Acc z = __shfl_sync(kFull, fz, gbase + q);
                if (c0 + q < deg) {  // slot order == ascending face id
                    total = dadd<Acc>(total, a);
                    wx = dadd<Acc>(wx, dmul<Acc>(a, x));
                    wy = dadd<Acc>(wy, dmul<Acc>(a, y));
                    wz = dadd<Acc>(wz, dmul<Acc>(a, z));
                }
            }
        }
        if (v >= 0 && glane == 0 && total > Acc(0)) T::store(p.work, v, total, wx, wy, wz);
    }
}

// Number of positions c, c + nc, c + 2 nc, ... that lie below `bound`.
__device__ __forceinline__ int owned_below(int bound, int c, int nc) { return bound > c ? (bound - c + nc - 1) / nc : 0; }

// Vertex ownership: CTA c owns the vertices at positions c, c + n_ctas, ...
// of `order`, so every dependency level (a contiguous run of `order`) is
// spread evenly over all CTAs and a CTA always updates the same vertices.
// With SMEM the CTA copies those vertices' incident-face slots into shared
// memory once; each wavefront step then only gathers positions from L2.
template <int MODE, int G, bool SMEM>
__global__ void __launch_bounds__(512) areal_sweeps_kernel(ArealParams p) {
    using T = Traits<MODE>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double stage_all[512 / 32][4][32];  // per-warp staging of face terms (float64 modes)
    double (*stage)[32] = stage_all[threadIdx.x >> 5];
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthreads = gridDim.x * blockDim.x;
    const int c = blockIdx.x;
    const int nc = gridDim.x;
    const int groups = blockDim.x / G;
    const int warp_first_group = (threadIdx.x >> 5) * (32 / G);
    const int my_group = (threadIdx.x & 31) / G;
    const int nloc = owned_below(p.n, c, nc);
    const int L = p.n_levels;
    const int D = p.stride;
    // shared-memory image (SMEM only): face slots, vertex ids and degrees of
    // the owned vertices, then per-level owned ranges and per-residue top level
    int4* ltri = reinterpret_cast<int4*>(smem);
    int* lvid = reinterpret_cast<int*>(ltri + (SMEM ? p.nloc_max * p.max_degree : 0));
    int* ldeg = lvid + p.nloc_max;
    int* lbeg = ldeg + p.nloc_max;
    int* lend = lbeg + L;
    int* hitop = lend + L;
    unsigned int phase = 0;
    int barrier_id = 0;

    if (SMEM) {
        for (int i = threadIdx.x; i < nloc; i += blockDim.x) {
            const int v = __ldg(p.order + c + i * nc);
            const int s0 = __ldg(p.slot_off + v);
            int d = __ldg(p.slot_off + v + 1) - s0;
            if (d < 0 || d > p.max_degree) {  // plan and max_degree disagree: report, stay inside the image
                if (atomicCAS(&p.ctl->status, CSG_OK, CSG_ERR_ARG) == CSG_OK) p.ctl->where = -3;
                d = 0;
            }
            lvid[i] = v;
            ldeg[i] = d;
            for (int j = 0; j < d; ++j) ltri[i * p.max_degree + j] = __ldg(p.slot_tri + s0 + j);
        }
        for (int l = threadIdx.x; l < L; l += blockDim.x) {
            lbeg[l] = owned_below(__ldg(p.level_begin + l), c, nc);
            lend[l] = owned_below(__ldg(p.level_end + l), c, nc);
        }
        for (int r = threadIdx.x; r < D; r += blockDim.x) hitop[r] = (L - 1) - ((L - 1 - r) % D + D) % D;
    }
    for (int v = tid; v < p.n; v += nthreads) T::pack(p.points, p.work, v);
    if (csg::grid_barrier(p.ctl, phase, p.timeout_ns, barrier_id++)) return;
    if (SMEM && csg::ld_relaxed_gpu(&p.ctl->status) != CSG_OK) return;  // a degree over max_degree: every CTA sees it

    const int last = p.iterations - 1;
    for (int start = 1; start <= last;) {
        int end = last;
        if (p.project_every > 0) end = min(last, ((start - 1) / p.project_every + 1) * p.project_every);
        const int S = end - start + 1;
        const int span = (S - 1) * D;        // host guarantees span + L < 2^31
        const int nsteps = span + L;
        int r = 0;                           // r == t mod D, kept incrementally
        for (int t = 0; t < nsteps; ++t, r = (r + 1 == D) ? 0 : r + 1) {
            // active levels: lo, lo + D, ..., hi (all congruent to t mod D)
            int hi, lo = t - span;
            if (lo < r) lo = r;
            int i0, i1;
            if (SMEM) {
                hi = t < L ? t : hitop[r];
                if (hi < lo) continue;  // no vertex of any sweep sits on this step
                i0 = lbeg[lo];
                i1 = lend[hi];
            } else {
                hi = t < L ? t : (L - 1) - ((L - 1 - r) % D + D) % D;
                if (hi < lo) continue;
                i0 = owned_below(__ldg(p.level_begin + lo), c, nc);
                i1 = owned_below(__ldg(p.level_end + hi), c, nc);
            }
            for (int base = i0 + warp_first_group; base < i1; base += groups) {
                const int i = base + my_group;
                int v = -1, deg = 0;
                const int4* tri = nullptr;
                if (i < i1) {
                    if (SMEM) {
                        v = lvid[i];
                        deg = ldeg[i];
                        tri = ltri + i * p.max_degree;
                    } else {
                        v = __ldg(p.order + c + i * nc);
                        const int s0 = __ldg(p.slot_off + v);
                        deg = __ldg(p.slot_off + v + 1) - s0;
                        tri = p.slot_tri + s0;
                    }
                }
                update_vertex<MODE, G, SMEM>(p, v, tri, deg, stage);
            }
            if (csg::grid_barrier(p.ctl, phase, p.timeout_ns, barrier_id++)) return;
        }
        if (p.project_every > 0 && end % p.project_every == 0) {
            for (int v = tid; v < p.n; v += nthreads) T::project(p.work, v, p.radius);
            if (csg::grid_barrier(p.ctl, phase, p.timeout_ns, barrier_id++)) return;
        }
        start = end + 1;
    }
    for (int v = tid; v < p.n; v += nthreads) T::unpack(p.work, p.points, v);
}

// ---------------------------------------------------------------------------
// Dataflow form of the sweeps (float32 storage modes).
//
// The grid barrier between wavefront steps is replaced by per-vertex versions.
// Each vertex is published as one 16-byte word (x, y, z, version), version = the
// number of sweeps the vertex has completed; a relaxed 16-byte load returns a
// position and the version it belongs to.  The words sit kWordPitch quads (64
// bytes) apart, so no two vertices' words share a 32-byte sector or its pair:
// polls of one vertex do not queue behind the publication of another (61,442
// vertices, 4,999 sweeps: 61.4 ms at 16 bytes, 53.9 at 32, 50.0 at 64 and at 128).
// Sweep s of vertex v needs lower-index neighbours at version s and
// higher-index neighbours and v itself at version s - 1, and neither can be
// further ahead: a lower neighbour u cannot finish sweep s + 1 before v
// finishes sweep s (v > u is its higher neighbour), a higher neighbour w cannot
// finish sweep s before v does.  So once every word shows its required version
// the values are exactly the sequential Gauss-Seidel inputs, and the group
// polls its faces' words until they do.  Each group walks the same wavefront
// order as the barrier form (step t, then its share of the step's vertices),
// which keeps progress guaranteed: the earliest unfinished update's inputs are
// all finished.  The projections ride in the wavefront too (a second array
// of projected words, written as each epoch's last sweep is published), so
// one wavefront runs every sweep and grid barriers remain only at the start
// and the end.
// Every wait is bounded: on timeout (or another CTA's failure) the kernel
// records the status and leaves.

using csg::ld_quad;
using csg::make_quad;
using csg::Quad;
using csg::quad_point;
using csg::quad_version;
using csg::st_quad;

// Ring of a vertex: itself, then the other vertices of its faces (at most
// 2 max_degree + 1 of them, the rows' capacity; the form is taken up to kRingMax);
// each face slot is coded as three ring indices (8 bits each).
constexpr int kRingMax = 20;

// Vertex v's published word is words[kWordPitch v], its projected word the quad
// kProjected further on (written once per projection epoch, so it may share the 64 bytes).
constexpr int kWordPitch = 4, kProjected = 2;

// Entries of a ring row and of a group's staged positions: one for every lane of the group at least.
__host__ __device__ inline int dataflow_ring_capacity(int max_degree, int lanes) {
    return 2 * max_degree + 1 > lanes ? 2 * max_degree + 1 : lanes;
}

// sweep mod project_every (> 0): a high multiply with the host's rounded-up reciprocal,
// exact while sweep * project_every < 2^32 (the host passes 0 when it may not be).
__device__ __forceinline__ unsigned int epoch_rest(const ArealParams& p, unsigned int sweep) {
    const unsigned int pe = static_cast<unsigned int>(p.project_every);
    if (p.epoch_magic == 0) return sweep % pe;
    return sweep - __umulhi(sweep, p.epoch_magic) * pe;
}

// Poll the words of ring members glane, glane + G, ... (`first` is this lane's member 0,
// -1 for none) until each shows the version this update needs (lower members sweep s, the
// others and the vertex itself s - 1), then stage their positions.  MEMBERS = 1 serves
// rings of at most G members (one word per lane).  `late` is kProjected in the sweep after
// a projection, whose previous-sweep members are the projected points.  A lane that has
// its version stops loading: the word cannot change before this update publishes, and each
// word a poll re-reads costs the SM's L1 data path a pass (with the shared-memory staging
// the kernel's busiest unit), which holds up the updates that could proceed.  For the same
// reason one poll is in flight per lane: two or three made the sweeps slower (77 and
// 99 ms against 62).  Returns false to abort.
template <int MEMBERS, int G>
__device__ __forceinline__ bool poll_ring(const ArealParams& p, const Quad* words, int late, int v, int first,
                                          const int* ring, int nring, unsigned int s, float4* pos) {
    const int glane = threadIdx.x & (G - 1);
    const Quad* from[MEMBERS];
    unsigned int need[MEMBERS];
    Quad w[MEMBERS];
#pragma unroll
    for (int q = 0; q < MEMBERS; ++q) {
        const int u = q == 0 ? first : (glane + q * G < nring ? ring[glane + q * G] : -1);
        need[q] = u < v ? s : s - 1;
        w[q] = Quad{0, static_cast<unsigned long long>(need[q]) << 32};  // no member: nothing to wait for
        from[q] = words + (static_cast<long long>(kWordPitch) * u + (u < v ? 0 : late));
        if (u >= 0) w[q] = ld_quad(from[q]);
    }
    unsigned int polls = 0;
    unsigned long long start = 0;
    while (true) {
        bool want = false;
#pragma unroll
        for (int q = 0; q < MEMBERS; ++q) want = want || quad_version(w[q]) != need[q];
        if (!__any_sync(kFull, want)) break;
        if (csg::warp_wait_expired(p.ctl, p.timeout_ns, polls, start)) return false;
#pragma unroll
        for (int q = 0; q < MEMBERS; ++q)
            if (quad_version(w[q]) != need[q]) w[q] = ld_quad(from[q]);
    }
#pragma unroll
    for (int q = 0; q < MEMBERS; ++q)
        if (q == 0 || glane + q * G < nring) pos[glane + q * G] = quad_point(w[q]);
    return true;
}

constexpr int kStagePitch = 34;  // doubles per staged row: the four rows of a warp start on different banks

// A warp's staged face terms (the float32 mode sums by shuffles).
template <int MODE>
__host__ __device__ constexpr int dataflow_stage_bytes() {
    return sizeof(typename Traits<MODE>::Acc) == 8 ? 4 * kStagePitch * static_cast<int>(sizeof(double)) : 0;
}

// The area total (lanes 0..2) and one coordinate's weighted sum (lane k: coordinate k) of up
// to G staged faces, added in slot order.  Slots past the last face hold +0, which leaves a
// sum that started from +0 unchanged, so the G additions need no test.
template <int G>
__device__ __forceinline__ void add_faces(const double (*stage)[kStagePitch], int glane, int gbase, double& total,
                                          double& wsum) {
    const double2* ta = reinterpret_cast<const double2*>(&stage[0][gbase]);
    const double2* tm = reinterpret_cast<const double2*>(&stage[1 + glane][gbase]);
#pragma unroll
    for (int q = 0; q < G / 2; ++q) {
        const double2 x = ta[q], y = tm[q];
        total = __dadd_rn(__dadd_rn(total, x.x), x.y);
        wsum = __dadd_rn(__dadd_rn(wsum, y.x), y.y);
    }
}

// One vertex update of sweep s by a group of G lanes (all 32 lanes call it;
// groups without an item pass v < 0 and nring = deg = 0).  The group polls the
// ring and stages the positions in shared memory (`pos`), then computes the
// faces exactly as update_vertex does (same arithmetic, slot order).  Lane 0
// publishes the point.  Returns false to abort.
template <int MODE, int G>
__device__ __forceinline__ bool update_vertex_df(const ArealParams& p, Quad* words, int v, const int* ring, int nring,
                                                 const int* code, int deg, unsigned int s,
                                                 double (*stage)[kStagePitch], float4* pos) {
    using T = Traits<MODE>;
    using Acc = typename T::Acc;
    using P3 = typename T::P3;
    const int lane = threadIdx.x & 31;
    const int glane = lane & (G - 1);
    const int gbase = lane & ~(G - 1);
    const int first = glane < nring ? ring[glane] : -1;
    // sweep s ends a projection epoch (publish the projected point too), or follows one
    bool at_end = false;
    int late = 0;
    if (p.project_every > 0) {
        const unsigned int rest = epoch_rest(p, s);
        at_end = rest == 0;
        if (s > 1 && (p.project_every == 1 || rest == 1)) late = kProjected;
    }
    const bool wide = __any_sync(kFull, max(nring, deg) > G);  // more ring members or faces than lanes in the warp
    if (!wide) {
        if (!poll_ring<1, G>(p, words, late, v, first, ring, nring, s, pos)) return false;
    } else {
        if (!poll_ring<(kRingMax + G - 1) / G, G>(p, words, late, v, first, ring, nring, s, pos)) return false;
    }
    __syncwarp();
    Acc total = 0, wx = 0, wy = 0, wz = 0;  // float path: every lane sums its group's faces
    double wsum = 0;                        // float64 path: lanes 0..2 sum one coordinate each
    auto corner = [&](int index) {
        const float4 q = pos[index & 255];
        return P3{q.x, q.y, q.z};
    };
    auto stage_face = [&](int j) {  // float64 path: face slot j's area and weighted centre
        double fa = 0, fx = 0, fy = 0, fz = 0;
        if (j < deg) {
            const int cd = code[j];
            Acc area, mx, my, mz;
            T::face(corner(cd), corner(cd >> 8), corner(cd >> 16), area, mx, my, mz);
            fa = area;
            fx = __dmul_rn(fa, mx);
            fy = __dmul_rn(fa, my);
            fz = __dmul_rn(fa, mz);
        }
        stage[0][lane] = fa;
        stage[1][lane] = fx;
        stage[2][lane] = fy;
        stage[3][lane] = fz;
        __syncwarp();
    };
    if constexpr (sizeof(Acc) == 8) {
        if (!wide) {
            stage_face(glane);
            if (glane < 3) add_faces<G>(stage, glane, gbase, total, wsum);
        } else {
            for (int c0 = 0; __any_sync(kFull, c0 < deg); c0 += G) {
                stage_face(c0 + glane);
                if (glane < 3) add_faces<G>(stage, glane, gbase, total, wsum);
                __syncwarp();
            }
        }
    } else {
        for (int c0 = 0; __any_sync(kFull, c0 < deg); c0 += G) {
            Acc fa = 0, fx = 0, fy = 0, fz = 0;
            if (c0 + glane < deg) {
                const int cd = code[c0 + glane];
                T::face(corner(cd), corner(cd >> 8), corner(cd >> 16), fa, fx, fy, fz);
            }
#pragma unroll
            for (int q = 0; q < G; ++q) {
                const Acc aa = __shfl_sync(kFull, fa, gbase + q);
                const Acc x = __shfl_sync(kFull, fx, gbase + q);
                const Acc y = __shfl_sync(kFull, fy, gbase + q);
                const Acc z = __shfl_sync(kFull, fz, gbase + q);
                if (c0 + q < deg) {  // slot order == ascending face id
                    total = dadd<Acc>(total, aa);
                    wx = dadd<Acc>(wx, dmul<Acc>(aa, x));
                    wy = dadd<Acc>(wy, dmul<Acc>(aa, y));
                    wz = dadd<Acc>(wz, dmul<Acc>(aa, z));
                }
            }
        }
    }
    // a vertex that does not move republishes its own position (ring member 0)
    float nx = 0.0f, ny = 0.0f, nz = 0.0f;
    if constexpr (sizeof(Acc) == 8) {
        float value = 0.0f;
        if (v >= 0 && glane < 3) {
            value = glane == 0 ? pos[0].x : (glane == 1 ? pos[0].y : pos[0].z);
            if (total > 0.0) {  // summed by each of lanes 0..2 (same order, same value)
                const double safe = total > 1.0e-20 ? total : 1.0e-20;
                value = __double2float_rn(__ddiv_rn(wsum, safe));
            }
        }
        nx = value;
        ny = __shfl_sync(kFull, value, gbase + 1);
        nz = __shfl_sync(kFull, value, gbase + 2);
    } else if (v >= 0 && glane == 0) {
        nx = pos[0].x;
        ny = pos[0].y;
        nz = pos[0].z;
        if (total > Acc(0)) {
            const float safe = total > 1.0e-20f ? total : 1.0e-20f;
            nx = __fdiv_rn(wx, safe);
            ny = __fdiv_rn(wy, safe);
            nz = __fdiv_rn(wz, safe);
        }
    }
    if (v >= 0 && glane == 0) {
        Quad* word = words + static_cast<long long>(kWordPitch) * v;
        st_quad(word, make_quad(nx, ny, nz, s));
        if (at_end) {
            // T::project_p3 of the float32 values just published, as a separate projection pass computes it
            const P3 q = T::project_p3(P3{nx, ny, nz}, p.radius);
            st_quad(word + kProjected, make_quad(q.x, q.y, q.z, s));
        }
    }
    __syncwarp();  // every lane is done with `pos` and `stage` before the next update overwrites them
    return true;
}

template <int MODE, int G>
__global__ void __launch_bounds__(512) areal_dataflow_kernel(ArealParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    Quad* words = static_cast<Quad*>(p.work);
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthreads = gridDim.x * blockDim.x;
    const int c = blockIdx.x;
    const int nc = gridDim.x;
    const int groups = blockDim.x / G;
    const int warp_first_group = (threadIdx.x >> 5) * (32 / G);
    const int my_group = (threadIdx.x & 31) / G;
    const int nloc = owned_below(p.n, c, nc);
    const int L = p.n_levels;
    const int D = p.stride;
    const int cap = dataflow_ring_capacity(p.max_degree, G);
    // shared-memory image: per warp the staged face terms; per group `cap` staged
    // positions; per owned vertex its description (id, degree | ring size << 8,
    // level / D), ring and face codes; per level the owned range; per residue the
    // top level
    double (*stage)[kStagePitch] = reinterpret_cast<double (*)[kStagePitch]>(smem) + 4 * (threadIdx.x >> 5);
    float4* pos0 = reinterpret_cast<float4*>(smem + (blockDim.x / 32) * dataflow_stage_bytes<MODE>());
    float4* pos = pos0 + (threadIdx.x / G) * cap;
    int4* lmeta = reinterpret_cast<int4*>(pos0 + (blockDim.x / G) * cap);
    int* lring = reinterpret_cast<int*>(lmeta + p.nloc_max);
    int* lcode = lring + p.nloc_max * cap;
    int* lbeg = lcode + p.nloc_max * p.max_degree;
    int* lend = lbeg + L;
    int* hitop = lend + L;
    unsigned int phase = 0;
    int barrier_id = 0;
    for (int l = threadIdx.x; l < L; l += blockDim.x) {
        const int b = owned_below(__ldg(p.level_begin + l), c, nc), e = owned_below(__ldg(p.level_end + l), c, nc);
        lbeg[l] = b;
        lend[l] = e;
        for (int i = b; i < e; ++i) lmeta[i].z = l / D;
    }
    for (int i = threadIdx.x; i < nloc; i += blockDim.x) {
        const int v = __ldg(p.order + c + i * nc);
        const int s0 = __ldg(p.slot_off + v);
        int d = __ldg(p.slot_off + v + 1) - s0;
        if (d < 0 || d > p.max_degree) {  // plan and max_degree disagree: report, stay inside the image
            if (atomicCAS(&p.ctl->status, CSG_OK, CSG_ERR_ARG) == CSG_OK) p.ctl->where = -3;
            d = 0;
        }
        int* ring = lring + i * cap;
        int nr = 1;
        ring[0] = v;
        for (int j = 0; j < d; ++j) {
            const int4 t = __ldg(p.slot_tri + s0 + j);
            const int u[3] = {t.x, t.y, t.z};
            int cd = 0;
            for (int k = 0; k < 3; ++k) {
                int at = 0;
                while (at < nr && ring[at] != u[k]) ++at;
                if (at == nr) {
                    if (nr == cap) {  // cannot be with at most max_degree faces round v; report, stay inside
                        if (atomicCAS(&p.ctl->status, CSG_OK, CSG_ERR_ARG) == CSG_OK) p.ctl->where = -1;
                        at = 0;
                    } else {
                        ring[nr++] = u[k];
                    }
                }
                cd |= at << (8 * k);
            }
            lcode[i * p.max_degree + j] = cd;
        }
        lmeta[i].x = v;
        lmeta[i].y = d | (nr << 8);
    }
    for (int r = threadIdx.x; r < D; r += blockDim.x) hitop[r] = (L - 1) - ((L - 1 - r) % D + D) % D;
    for (int v = tid; v < p.n; v += nthreads) {
        const float* q = static_cast<const float*>(p.points) + 3LL * v;
        Quad* word = words + static_cast<long long>(kWordPitch) * v;
        st_quad(word, make_quad(q[0], q[1], q[2], 0u));
        // projected words start at version 0, below any epoch's end: a word left
        // from an earlier call on the same scratch never satisfies a poll
        st_quad(word + kProjected, make_quad(0.0f, 0.0f, 0.0f, 0u));
    }
    if (csg::grid_barrier(p.ctl, phase, p.timeout_ns, barrier_id++)) return;
    // a ring overflow or a degree over max_degree: the same answer in every CTA
    if (csg::ld_relaxed_gpu(&p.ctl->status) != CSG_OK) return;

    // One wavefront over every sweep.  The projection after sweep b (b a multiple of
    // project_every) is applied by each vertex's group as it publishes sweep b, into
    // its projected word; the updates of sweep b + 1 read their previous-sweep
    // members (higher neighbours and the vertex itself) from there, the updates of
    // sweep b read the unprojected words.  The wavefront therefore
    // never drains at a projection.
    const int last = p.iterations - 1;
    if (last >= 1) {
        const int span = (last - 1) * D;  // host guarantees span + L < 2^31
        const int nsteps = span + L;
        int r = 0, tq = 0;                // t mod D, t / D
        for (int t = 0; t < nsteps; ++t) {
            int lo = t - span;
            if (lo < r) lo = r;
            const int hi = t < L ? t : hitop[r];
            if (hi >= lo) {
                const int i0 = lbeg[lo], i1 = lend[hi];
                for (int base = i0 + warp_first_group; base < i1; base += groups) {
                    const int i = base + my_group;
                    int4 m = make_int4(-1, 0, 0, 0);
                    if (i < i1) m = lmeta[i];
                    const unsigned int sweep = static_cast<unsigned int>(1 + tq - m.z);  // t and the level agree mod D
                    if (!update_vertex_df<MODE, G>(p, words, m.x, lring + i * cap, m.y >> 8,
                                                   lcode + i * p.max_degree, m.y & 255, sweep, stage, pos))
                        return;
                }
            }
            if (++r == D) {
                r = 0;
                ++tq;
            }
        }
    }
    if (csg::grid_barrier(p.ctl, phase, p.timeout_ns, barrier_id++)) return;
    const int result = (p.project_every > 0 && last >= 1 && last % p.project_every == 0) ? kProjected : 0;
    for (int v = tid; v < p.n; v += nthreads) {
        float* q = static_cast<float*>(p.points) + 3LL * v;
        const float4 x = quad_point(ld_quad(words + static_cast<long long>(kWordPitch) * v + result));
        q[0] = x.x;
        q[1] = x.y;
        q[2] = x.z;
    }
}

constexpr size_t kMaxTopologySmem = 200 * 1024;
constexpr size_t kMaxDataflowSmem = 216 * 1024;  // the staged face terms are part of it

template <int MODE, int G>
int launch(ArealParams params, int n_ctas, int threads, cudaStream_t stream) {
    int device = 0, sms = 0;
    CSG_CUDA_CHECK(cudaGetDevice(&device));
    CSG_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    if (n_ctas <= 0) n_ctas = sms;
    params.nloc_max = (params.n + n_ctas - 1) / n_ctas;
    void* args[] = {&params};
    bool launched = false;
    // The dataflow form, the barrier form with its topology in shared memory, and from global memory: the first
    // whose CTAs fit the device together.
    if constexpr (MODE != CSG_ARITH_FP64) {
        // a ring has at most 2 max_degree + 1 vertices
        if (params.allow_dataflow && params.max_degree > 0 && 2 * params.max_degree + 1 <= kRingMax) {
            const long long pe = params.project_every;
            params.epoch_magic = pe > 1 && pe * params.iterations < (1LL << 32)
                                     ? static_cast<unsigned int>(((1LL << 32) + pe - 1) / pe)
                                     : 0u;
            const size_t cap = dataflow_ring_capacity(params.max_degree, G);
            const size_t smem = (threads / 32) * dataflow_stage_bytes<MODE>() + sizeof(float4) * (threads / G) * cap +
                                static_cast<size_t>(params.nloc_max) * sizeof(int) * (cap + params.max_degree + 4) +
                                sizeof(int) * (2 * static_cast<size_t>(params.n_levels) + params.stride);
            if (smem <= kMaxDataflowSmem) {
                const int rc = csg::launch_if_resident(reinterpret_cast<const void*>(areal_dataflow_kernel<MODE, G>), n_ctas,
                                                       threads, smem, args, stream, launched);
                if (rc || launched) return rc;
            }
        }
    }
    const size_t smem = static_cast<size_t>(params.nloc_max) * (params.max_degree * sizeof(int4) + 2 * sizeof(int)) +
                        sizeof(int) * (2 * static_cast<size_t>(params.n_levels) + params.stride);
    if (params.max_degree > 0 && smem <= kMaxTopologySmem) {
        const int rc = csg::launch_if_resident(reinterpret_cast<const void*>(areal_sweeps_kernel<MODE, G, true>), n_ctas,
                                               threads, smem, args, stream, launched);
        if (rc || launched) return rc;
    }
    const int rc = csg::launch_if_resident(reinterpret_cast<const void*>(areal_sweeps_kernel<MODE, G, false>), n_ctas,
                                           threads, 0, args, stream, launched);
    if (rc || launched) return rc;
    return csg::fail(CSG_ERR_LAUNCH, "areal sweeps: %d CTAs x %d threads cannot be co-resident on %d SMs", n_ctas, threads, sms);
}

template <int MODE>
int dispatch_lanes(const ArealParams& params, int n_ctas, int threads, int lanes, cudaStream_t stream) {
    switch (lanes) {
        case 4: return launch<MODE, 4>(params, n_ctas, threads, stream);
        case 8: return launch<MODE, 8>(params, n_ctas, threads, stream);
        case 16: return launch<MODE, 16>(params, n_ctas, threads, stream);
        default: return csg::fail(CSG_ERR_ARG, "lanes_per_vertex must be 4, 8 or 16 (got %d)", lanes);
    }
}

size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

// Barrier whose expected arrival count is one more than the grid holds: the
// bounded wait must give up and record CSG_ERR_TIMEOUT.
__global__ void k_div3_selftest(const double* __restrict__ x, long long n, double* __restrict__ a,
                                double* __restrict__ b) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    a[i] = __ddiv_rn(x[i], 3.0);
    b[i] = csg::div3_rn(x[i]);
}

__global__ void barrier_timeout_selftest_kernel(csg::Control* ctl, unsigned long long timeout_ns) {
    unsigned int phase = 1;
    csg::grid_barrier(ctl, phase, timeout_ns, 1);
}

}  // namespace

extern "C" {

size_t csg_areal_scratch_bytes(int n_vertices, int arithmetic) {
    if (n_vertices < 1 || (arithmetic != CSG_ARITH_CAT && arithmetic != CSG_ARITH_FP32 && arithmetic != CSG_ARITH_FP64))
        return 0;
    // float64: a double4 working copy; float32 modes: the dataflow form's kWordPitch
    // quads per vertex (the barrier form uses the first 16 bytes per vertex)
    return sizeof(csg::Control) + align256(64 * static_cast<size_t>(n_vertices));
}

int csg_areal_sweeps(void* points, int n_vertices, const int32_t* slot_off, const int32_t* slot_tri,
                     const int32_t* order, const int32_t* level_begin, const int32_t* level_end, int n_levels,
                     int level_stride, int max_degree, int iterations, int project_every, double radius, int arithmetic, void* scratch,
                     size_t scratch_bytes, int n_ctas, int threads_per_cta, int lanes_per_vertex, double timeout_s,
                     csg_stream_t stream) {
    if (!points || n_vertices < 1 || !slot_off || !slot_tri || !order || !level_begin || !level_end || !scratch)
        return csg::fail(CSG_ERR_ARG, "areal sweeps: null pointer or empty mesh");
    if (n_levels < 1 || n_levels > n_vertices || level_stride < 1 || iterations < 1 || project_every < 0 ||
        max_degree < 0)
        return csg::fail(CSG_ERR_ARG, "areal sweeps: bad schedule (levels %d, stride %d, iterations %d, project %d)",
                         n_levels, level_stride, iterations, project_every);
    {
        const long long sweeps_per_epoch = project_every > 0 ? project_every : iterations;
        if ((sweeps_per_epoch - 1) * static_cast<long long>(level_stride) + n_levels >= (1LL << 31))
            return csg::fail(CSG_ERR_ARG, "areal sweeps: wavefront epoch longer than 2^31 steps");
    }
    if (arithmetic < CSG_ARITH_CAT || arithmetic > CSG_ARITH_FP64)
        return csg::fail(CSG_ERR_ARG, "areal sweeps: unknown arithmetic %d", arithmetic);
    if (scratch_bytes < csg_areal_scratch_bytes(n_vertices, arithmetic))
        return csg::fail(CSG_ERR_ARG, "areal sweeps: scratch %zu bytes < required %zu", scratch_bytes,
                         csg_areal_scratch_bytes(n_vertices, arithmetic));
    if (reinterpret_cast<uintptr_t>(scratch) % 256 != 0 || reinterpret_cast<uintptr_t>(slot_tri) % 16 != 0)
        return csg::fail(CSG_ERR_ARG, "areal sweeps: scratch must be 256-byte and slot_tri 16-byte aligned");
    if (threads_per_cta <= 0) threads_per_cta = 512;
    if (lanes_per_vertex <= 0) lanes_per_vertex = 8;
    if (threads_per_cta % 32 != 0 || threads_per_cta > 512)
        return csg::fail(CSG_ERR_ARG, "areal sweeps: threads_per_cta must be a multiple of 32 up to 512");
    if (timeout_s <= 0.0) timeout_s = 2.0;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    ArealParams p{};
    p.points = points;
    p.ctl = static_cast<csg::Control*>(scratch);
    p.work = static_cast<char*>(scratch) + sizeof(csg::Control);
    p.slot_tri = reinterpret_cast<const int4*>(slot_tri);
    p.slot_off = slot_off;
    p.order = order;
    p.level_begin = level_begin;
    p.level_end = level_end;
    p.n = n_vertices;
    p.n_levels = n_levels;
    p.stride = level_stride;
    p.max_degree = max_degree;
    p.iterations = iterations;
    p.project_every = project_every;
    p.allow_dataflow = 1;
    p.radius = radius;
    p.timeout_ns = static_cast<unsigned long long>(timeout_s * 1e9);
    CSG_CUDA_CHECK(cudaMemsetAsync(scratch, 0, sizeof(csg::Control), s));
    switch (arithmetic) {
        case CSG_ARITH_CAT: return dispatch_lanes<CSG_ARITH_CAT>(p, n_ctas, threads_per_cta, lanes_per_vertex, s);
        case CSG_ARITH_FP32: return dispatch_lanes<CSG_ARITH_FP32>(p, n_ctas, threads_per_cta, lanes_per_vertex, s);
        default: return dispatch_lanes<CSG_ARITH_FP64>(p, n_ctas, threads_per_cta, lanes_per_vertex, s);
    }
}

int csg_selftest_div3(const double* x, long long n, double* by_division, double* by_multiplies, csg_stream_t stream) {
    if (!x || n < 0 || !by_division || !by_multiplies) return csg::fail(CSG_ERR_ARG, "div3 self-test: bad arguments");
    if (n == 0) return CSG_OK;
    (csg::note_launch(), k_div3_selftest<<<static_cast<unsigned>((n + 255) / 256), 256, 0,
                                          reinterpret_cast<cudaStream_t>(stream)>>>(x, n, by_division, by_multiplies));
    CSG_CUDA_CHECK(cudaGetLastError());
    return CSG_OK;
}

int csg_selftest_barrier_timeout(void* scratch, size_t scratch_bytes, double timeout_s, csg_stream_t stream) {
    if (!scratch || scratch_bytes < sizeof(csg::Control) || timeout_s <= 0.0 || timeout_s > 10.0)
        return csg::fail(CSG_ERR_ARG, "barrier self-test: need 256 bytes of scratch and 0 < timeout_s <= 10");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    csg::Control* ctl = static_cast<csg::Control*>(scratch);
    unsigned long long timeout_ns = static_cast<unsigned long long>(timeout_s * 1e9);
    CSG_CUDA_CHECK(cudaMemsetAsync(scratch, 0, sizeof(csg::Control), s));
    void* args[] = {&ctl, &timeout_ns};
    CSG_CUDA_CHECK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(barrier_timeout_selftest_kernel), dim3(2),
                                               dim3(32), args, 0, s));
    csg::note_launch();
    return CSG_OK;
}

int csg_read_status(const void* scratch, csg_stream_t stream, int* status, int* where) {
    if (!scratch || !status) return csg::fail(CSG_ERR_ARG, "read_status: null pointer");
    csg::Control ctl{};
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    CSG_CUDA_CHECK(cudaMemcpyAsync(&ctl, scratch, sizeof(ctl), cudaMemcpyDeviceToHost, s));
    CSG_CUDA_CHECK(cudaStreamSynchronize(s));
    *status = ctl.status;
    if (where) *where = ctl.where;
    return CSG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free variant of csg_areal_sweeps.
//
// Some callers cannot call cudaMalloc: code that runs while a CUDA stream
// capture is active on its thread (cudaMalloc is refused in the default
// capture mode), hosts that hand all device memory to their own pool
// allocator up front, and thin foreign-function bindings that pass device
// pointers they were given but own no device allocator.  For them the sweep
// kernel's working memory (the 256-byte control block and the float4 /
// double4 position working copy) lives in the file-scope array below, which
// every GPU that loads this library holds until the process exits.
// Limits: 262,144 vertices in the float32 modes, 131,072 in float64 mode.

namespace {
constexpr size_t kNoAllocWorkBytes = static_cast<size_t>(262144) * sizeof(float4);  // 4 MiB
constexpr size_t kNoAllocBytes = sizeof(csg::Control) + kNoAllocWorkBytes;
}  // namespace

static __device__ __align__(256) unsigned char g_areal_noalloc_scratch[kNoAllocBytes];

namespace {
std::mutex g_noalloc_mutex;
constexpr int kNoAllocMaxDevices = 64;
void* g_noalloc_address[kNoAllocMaxDevices] = {};

// Device address of g_areal_noalloc_scratch on the current device, looked up
// once per device (the name itself is only a host-side stand-in).  The cached
// address belongs to the device's primary context: after cudaDeviceReset the
// module may load elsewhere, so this entry point must not be used across a
// device reset.
int noalloc_scratch(void** out) {
    int device = 0;
    CSG_CUDA_CHECK(cudaGetDevice(&device));
    if (device < 0 || device >= kNoAllocMaxDevices)
        return csg::fail(CSG_ERR_UNSUPPORTED, "areal sweeps (no-alloc): device ordinal %d >= %d", device,
                         kNoAllocMaxDevices);
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_address[device] == nullptr) {
        void* address = nullptr;
        const cudaError_t err = cudaGetSymbolAddress(&address, g_areal_noalloc_scratch);
        if (err != cudaSuccess || address == nullptr)
            return csg::fail(CSG_ERR_CUDA, "areal sweeps (no-alloc): cudaGetSymbolAddress failed: %s",
                             cudaGetErrorString(err));
        g_noalloc_address[device] = address;
    }
    *out = g_noalloc_address[device];
    return CSG_OK;
}
}  // namespace

extern "C" int csg_areal_sweeps_noalloc(void* points, int n_vertices, const int32_t* slot_off, const int32_t* slot_tri,
                                        const int32_t* order, const int32_t* level_begin, const int32_t* level_end,
                                        int n_levels, int level_stride, int max_degree, int iterations,
                                        int project_every, double radius, int arithmetic, int n_ctas,
                                        int threads_per_cta, int lanes_per_vertex, double timeout_s,
                                        int* status_out, csg_stream_t stream) {
    if (!points || n_vertices < 1 || !slot_off || !slot_tri || !order || !level_begin || !level_end)
        return csg::fail(CSG_ERR_ARG, "areal sweeps (no-alloc): null pointer or empty mesh");
    if (arithmetic < CSG_ARITH_CAT || arithmetic > CSG_ARITH_FP64)
        return csg::fail(CSG_ERR_ARG, "areal sweeps (no-alloc): unknown arithmetic %d", arithmetic);
    // the barrier form: a float4 (float32 modes) or double4 working copy
    const size_t need = sizeof(csg::Control) +
                        align256((arithmetic == CSG_ARITH_FP64 ? sizeof(D4) : sizeof(float4)) *
                                 static_cast<size_t>(n_vertices));
    if (need > kNoAllocBytes)
        return csg::fail(CSG_ERR_ARG,
                         "areal sweeps (no-alloc): %d vertices need %zu bytes of working memory, more than the "
                         "built-in %zu (at most %d vertices in float32 modes, %d in float64 mode)",
                         n_vertices, need, kNoAllocBytes, 262144, 131072);
    if (n_levels < 1 || n_levels > n_vertices || level_stride < 1 || iterations < 1 || project_every < 0 ||
        max_degree < 0)
        return csg::fail(CSG_ERR_ARG, "areal sweeps (no-alloc): bad schedule (levels %d, stride %d, iterations %d)",
                         n_levels, level_stride, iterations);
    {
        const long long sweeps_per_epoch = project_every > 0 ? project_every : iterations;
        if ((sweeps_per_epoch - 1) * static_cast<long long>(level_stride) + n_levels >= (1LL << 31))
            return csg::fail(CSG_ERR_ARG, "areal sweeps (no-alloc): wavefront epoch longer than 2^31 steps");
    }
    if (reinterpret_cast<uintptr_t>(slot_tri) % 16 != 0)
        return csg::fail(CSG_ERR_ARG, "areal sweeps (no-alloc): slot_tri must be 16-byte aligned");
    if (threads_per_cta <= 0) threads_per_cta = 512;
    if (lanes_per_vertex <= 0) lanes_per_vertex = 8;
    if (threads_per_cta % 32 != 0 || threads_per_cta > 512)
        return csg::fail(CSG_ERR_ARG, "areal sweeps (no-alloc): threads_per_cta must be a multiple of 32 up to 512");
    if (timeout_s <= 0.0) timeout_s = 2.0;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (status_out != nullptr) {
        // reading the status back waits for the kernel, which a stream being captured cannot do
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        CSG_CUDA_CHECK(cudaStreamIsCapturing(s, &capture));
        if (capture != cudaStreamCaptureStatusNone)
            return csg::fail(CSG_ERR_ARG, "areal sweeps (no-alloc): status_out must be NULL while the stream is "
                                          "being captured");
    }
    void* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    ArealParams p{};
    p.points = points;
    p.ctl = static_cast<csg::Control*>(scratch);
    p.work = static_cast<char*>(scratch) + sizeof(csg::Control);
    p.slot_tri = reinterpret_cast<const int4*>(slot_tri);
    p.slot_off = slot_off;
    p.order = order;
    p.level_begin = level_begin;
    p.level_end = level_end;
    p.n = n_vertices;
    p.n_levels = n_levels;
    p.stride = level_stride;
    p.max_degree = max_degree;
    p.iterations = iterations;
    p.project_every = project_every;
    p.radius = radius;
    p.timeout_ns = static_cast<unsigned long long>(timeout_s * 1e9);
    // The array keeps the previous call's contents: the control block (barrier
    // counter and status) must start at zero; the working copy is fully
    // rewritten from `points` by the kernel itself.
    CSG_CUDA_CHECK(cudaMemsetAsync(scratch, 0, sizeof(csg::Control), s));
    switch (arithmetic) {
        case CSG_ARITH_CAT: rc = dispatch_lanes<CSG_ARITH_CAT>(p, n_ctas, threads_per_cta, lanes_per_vertex, s); break;
        case CSG_ARITH_FP32: rc = dispatch_lanes<CSG_ARITH_FP32>(p, n_ctas, threads_per_cta, lanes_per_vertex, s); break;
        default: rc = dispatch_lanes<CSG_ARITH_FP64>(p, n_ctas, threads_per_cta, lanes_per_vertex, s); break;
    }
    if (rc || status_out == nullptr) return rc;
    csg::Control ctl{};
    CSG_CUDA_CHECK(cudaMemcpyAsync(&ctl, scratch, sizeof(ctl), cudaMemcpyDeviceToHost, s));
    CSG_CUDA_CHECK(cudaStreamSynchronize(s));
    *status_out = ctl.status;
    if (ctl.status != CSG_OK)
        return csg::fail(ctl.status, "areal sweeps (no-alloc): kernel reported status %d at barrier %d", ctl.status,
                         ctl.where);
    return CSG_OK;
}
