// el_advect.cu -- semi-Lagrangian advection of the level set and the MAC velocity.
//
// Reference: src/project/3d/fluid/advection.cpp:9-27 (loop drivers), include/nama/math/ode.h
// (StaggeredGridField, trace_rk2), include/nama/math/interpolation.h (lerp, weno6_interp).
// Per output sample: sample position -> backtrace through the old velocity (trilinear MAC
// interpolation at every RK stage) -> trilinear or WENO6 sample of the old field at the foot
// point.  Two forms: advect_kernel, one thread per sample reading global memory (a field other than
// the advecting velocity on a face grid; WENO6 face samples), and the tiled kernels below, which
// stage what a tile of samples reads (the velocity boxes; for WENO6 the level-set box and its x-pass
// smoothness terms) in shared memory once -- under the CFL limit the foot point moves at most about
// one cell -- and fall back to the global reads for a sample whose stencil leaves the box.  The
// boxes arrive by TMA box copies (cp.async.bulk.tensor) wherever the array's row pitch is a multiple
// of 16 bytes; the parts of a box outside the grid are then filled in from the clamped entries in
// shared memory, so that a box holds the clamped grid either way.
#include <cstring>
#include <limits>
#include <type_traits>

#include "el_div.cuh"
#include "el_internal.cuh"
#include "el_tma.cuh"

namespace el {

template <typename T>
struct Mac {
    GridView<T> u, v, w;
};

struct DtArg {
    const Scalars* s;  // device scalars holding dt, or null
    double v;          // dt by value when s is null
};

__device__ __forceinline__ double dt_value(const DtArg& a) { return a.s ? a.s->dt : a.v; }

// Set when a wait for a tile's box copies of a context's advection gave up (the tile's outputs are then
// NaN, so that the step's solve fails on them); read and cleared by advect_fault_take().  The stateless
// operators, which no context's solve follows, leave the NaN alone (BoxMap::on 2).
__device__ unsigned advect_wait_fault;

// a box copy of one array (on: BoxCopies; BOX_NONE: the array is staged by plain loads)
struct BoxMap {
    CUtensorMap m;
    int on;
};
struct MacMaps {
    BoxMap c[3];
};

// Positions.  A face sample's backtrace (and an FP64 cell's) is kept as its displacement in cells,
// relative to the sample itself: the RK stages are d = -(dt / dx) (weights . velocities), and a read at a displaced
// position takes the floor and the fraction of the displacement per axis (plus the half cell
// between cell and face samples).  Against absolute positions this leaves out, per coordinate, two
// subtractions and a product (FP32) or a division (FP64: fifteen divisions a velocity sample,
// nine FP64 operations each), and the fraction carries the rounding of a number near 1, not of a
// coordinate of hundreds of cells.
//
// h: -1/2 along the sample's own face axis, 0 along the others and for cell samples; a position
// d cells away has the coordinate d + h among cell-type samples and d + h + 1/2 among face-type
// ones, relative to the sample's index.
//
// The FP32 level set keeps absolute positions, (x - origin - dx / 2) / dx, as the reference's loops:
// the ghost-fluid fractions of the projection divide by distances to the surface down to a
// hundredth of a cell, so that another rounding of the positions, a more exact one too, shows in
// the projected velocity a thousand times larger.

// floor(e) and e - floor(e).  FP64: within two cells, where every stage of a step under the CFL limit
// lies, by comparisons of the bits (a floor and its conversion are FP64-pipe operations).  -0 has floor 0
// and -1 floor -1, both with fraction 0: a sample at rest is displaced by -dt / dx * 0 = -0 and keeps
// its value whatever its neighbours hold.  FP32: e + 1.5 * 2^23 rounded toward -inf holds floor(e) in
// its low mantissa bits (exact for |e| < 2^22); outside that range (and for NaN) the index lands
// millions of cells away, i.e. outside every staged box and grid, and the sample takes the general path.
template <typename T>
__device__ __forceinline__ void floor_index(T e, int& idx, T& frac) {
    if constexpr (sizeof(T) == 4) {
        const float big = 12582912.0f;  // 1.5 * 2^23, bit pattern 0x4B400000
        const float r = __fadd_rd(e, big);
        idx = (int)((unsigned)__float_as_int(r) - 0x4B400000u);
        frac = e - (r - big);
    } else {
        const unsigned long long bits = (unsigned long long)__double_as_longlong(e);
        if ((bits & 0x7fffffffffffffffull) < 0x4000000000000000ull) {
            const bool neg = bits > 0x8000000000000000ull;
            const bool far = neg ? bits > 0xbff0000000000000ull : (bits & 0x7fffffffffffffffull) >= 0x3ff0000000000000ull;
            idx = neg ? (far ? -2 : -1) : (far ? 1 : 0);
            frac = e - __hiloint2double(neg ? (far ? (int)0xc0000000 : (int)0xbff00000) : (far ? 0x3ff00000 : 0), 0);
        } else {
            const T fl = floor(e);
            idx = (int)fl;
            frac = e - fl;
        }
    }
}

// One axis of a position: floor indices and fractions among cell-type and face-type samples.
template <typename T>
struct AxisCF {
    int c, f;
    T wc, wf;
};

// FP32: both floors in packed arithmetic (lane .x cell, .y face), as floor_index, plus base
__device__ __forceinline__ AxisCF<float> axis_floor(float2 e, int base) {
    const float big = 12582912.0f;
    const float2 r = __fadd2_rd(e, make_float2(big, big));
    const float2 fl = __fadd2_rn(r, make_float2(-big, -big));
    const float2 w = __ffma2_rn(fl, make_float2(-1.f, -1.f), e);  // e - fl
    const unsigned b = (unsigned)base - 0x4B400000u;
    return AxisCF<float>{(int)((unsigned)__float_as_int(r.x) + b), (int)((unsigned)__float_as_int(r.y) + b), w.x, w.y};
}

// d cells away from sample index i
template <typename T>
__device__ __forceinline__ AxisCF<T> axis_rel(int i, T d, T h) {
    if constexpr (sizeof(T) == 4) {
        return axis_floor(__fadd2_rn(make_float2(d, d), make_float2(h, h + 0.5f)), i);
    } else {
        AxisCF<T> a;
        floor_index(h == T(0) ? d : d + h, a.c, a.wc);
        floor_index(h == T(0) ? d + T(0.5) : d, a.f, a.wf);
        a.c = (int)((unsigned)a.c + (unsigned)i);
        a.f = (int)((unsigned)a.f + (unsigned)i);
        return a;
    }
}

// the cell and face coordinates of an absolute FP32 position: (x - origin - dx / 2) / dx with the
// origins 0 (cells) and -dx / 2 (faces)
__device__ __forceinline__ float2 coord_abs(float x, float dx, float inv_dx) {
    const float q = 0.5f * dx;
    return __fmul2_rn(__fadd2_rn(__fadd2_rn(make_float2(x, x), make_float2(-0.f, q)), make_float2(-q, -q)),
                      make_float2(inv_dx, inv_dx));
}

template <typename T>
struct Vec3T {
    T x, y, z;
};

template <typename T>
struct Axes {
    AxisCF<T> x, y, z;
};
template <typename T>
__device__ __forceinline__ Axes<T> axes_rel(int i, int j, int k, const Vec3T<T>& h, const Vec3T<T>& d) {
    return Axes<T>{axis_rel(i, d.x, h.x), axis_rel(j, d.y, h.y), axis_rel(k, d.z, h.z)};
}
__device__ __forceinline__ Axes<float> axes_abs(const Vec3T<float>& p, float dx, float inv_dx) {
    return Axes<float>{axis_floor(coord_abs(p.x, dx, inv_dx), 0), axis_floor(coord_abs(p.y, dx, inv_dx), 0),
                       axis_floor(coord_abs(p.z, dx, inv_dx), 0)};
}

// flat index of a sample; 32 bits hold it (every grid has fewer than 2^31 samples), and 64-bit
// products cost several integer instructions each
template <typename T>
__device__ __forceinline__ int cell_index(const GridView<T>& g, int i, int j, int k) {
    return i + g.n0 * (j + g.n1 * k);
}

// the 8 points of a trilinear read at floor indices (i, j, k) are inside the grid (then clamping
// changes none of them)
template <typename T>
__device__ __forceinline__ bool tri_inside(const GridView<T>& g, int i, int j, int k) {
    return (unsigned)i < (unsigned)(g.n0 - 1) && (unsigned)j < (unsigned)(g.n1 - 1) && (unsigned)k < (unsigned)(g.n2 - 1);
}

// the trilinear combination of 8 loaded points: x, then y, then z lerps; FP32 with the z = 0 and
// z = 1 halves side by side in packed float2 arithmetic.  ZF: the form of its z lerp (LerpForm).
template <typename T, int ZF = LERP_ANY>
__device__ __forceinline__ T tri_mix(T fx, T fy, T fz, T c000, T c100, T c010, T c110, T c001, T c101, T c011,
                                     T c111) {
    if constexpr (sizeof(T) == 4) {
        auto lerp2 = [](float2 a, float2 b, float f) {
            const float g = 1.f - f;
            return __ffma2_rn(make_float2(f, f), b, __fmul2_rn(make_float2(g, g), a));
        };
        const float2 x0 = lerp2(make_float2(c000, c001), make_float2(c100, c101), fx);
        const float2 x1 = lerp2(make_float2(c010, c011), make_float2(c110, c111), fx);
        const float2 y = lerp2(x0, x1, fy);
        return lerp_form<ZF>(y.x, y.y, fz);
    } else {
        return tri_combine(fx, fy, fz, c000, c100, c010, c110, c001, c101, c011, c111);
    }
}

// the 8 values of an inside read: one base address and fixed strides
template <typename T>
struct Tri8 {
    T c[8];
};
template <typename T>
__device__ __forceinline__ Tri8<T> tri_load(const GridView<T>& g, int i, int j, int k) {
    const T* p = g.d + cell_index(g, i, j, k);
    const T *q = p + g.n0, *r = p + g.n0 * g.n1, *t = r + g.n0;
    return Tri8<T>{{__ldg(p), __ldg(p + 1), __ldg(q), __ldg(q + 1), __ldg(r), __ldg(r + 1), __ldg(t), __ldg(t + 1)}};
}
template <typename T>
__device__ __forceinline__ T tri_mix(const Tri8<T>& v, T fx, T fy, T fz) {
    return tri_mix(fx, fy, fz, v.c[0], v.c[1], v.c[2], v.c[3], v.c[4], v.c[5], v.c[6], v.c[7]);
}

// trilinear read of the sample's own grid, d cells away from sample (i, j, k)
template <typename T, bool TILED>
__device__ __forceinline__ T own_at(const GridView<T>& g, int i, int j, int k, const Vec3T<T>& d) {
    int bi, bj, bk;
    T fx, fy, fz;
    floor_index(d.x, bi, fx);
    floor_index(d.y, bj, fy);
    floor_index(d.z, bk, fz);
    bi = (int)((unsigned)bi + (unsigned)i);
    bj = (int)((unsigned)bj + (unsigned)j);
    bk = (int)((unsigned)bk + (unsigned)k);
    // FP32: the forms are part of the level set's rounding (level_set_foot)
    constexpr int X10 = sizeof(T) == 8 ? LERP_ANY : (TILED ? LERP_B : LERP_A);
    constexpr int X00 = sizeof(T) == 8 ? LERP_ANY : LERP_A, R = sizeof(T) == 8 ? LERP_ANY : LERP_B;
    if (tri_inside(g, bi, bj, bk)) {
        const Tri8<T> v = tri_load(g, bi, bj, bk);
        return tri_combine<X00, X10, R>(fx, fy, fz, v.c[0], v.c[1], v.c[2], v.c[3], v.c[4], v.c[5], v.c[6], v.c[7]);
    }
    return tri_clamped<X00, X10, R>(g, i, j, k, d.x, d.y, d.z);
}

// The clamped gathers of u, v, w for a position outside the grid (or a box): d cells away from sample
// (i, j, k), or at an absolute position.
template <typename T>
struct FarRel {
    int i, j, k;
    Vec3T<T> h, d;
    template <int C>
    __device__ __forceinline__ T at(const GridView<T>& g) const {
        const T q = T(0.5);
        return tri_clamped(g, i, j, k, d.x + (h.x + (C == 0 ? q : T(0))), d.y + (h.y + (C == 1 ? q : T(0))),
                           d.z + (h.z + (C == 2 ? q : T(0))));
    }
};
struct FarAbs {
    Vec3T<float> p;
    float dx, inv_dx;
    template <int C>
    __device__ __forceinline__ float at(const GridView<float>& g) const {
        const float2 x = coord_abs(p.x, dx, inv_dx), y = coord_abs(p.y, dx, inv_dx), z = coord_abs(p.z, dx, inv_dx);
        return tri_clamped(g, 0, 0, 0, C == 0 ? x.y : x.x, C == 1 ? y.y : y.x, C == 2 ? z.y : z.x);
    }
};

// u, v, w at one position from global memory: the three components share six axis coordinates (u at
// a face in x, cells in y and z; v and w likewise).  When all three reads are inside the grid (the
// common case) their 24 loads go out together from fixed offsets; otherwise each takes the
// clamped gather -- the same values either way
template <typename T, typename FAR>
__device__ __forceinline__ Vec3T<T> velocity_global(const Mac<T>& m, const Axes<T>& a, const FAR& far) {
    const AxisCF<T>&x = a.x, &y = a.y, &z = a.z;
    if (tri_inside(m.u, x.f, y.c, z.c) && tri_inside(m.v, x.c, y.f, z.c) && tri_inside(m.w, x.c, y.c, z.f)) {
        const Tri8<T> u = tri_load(m.u, x.f, y.c, z.c), v = tri_load(m.v, x.c, y.f, z.c), w = tri_load(m.w, x.c, y.c, z.f);
        return Vec3T<T>{tri_mix(u, x.wf, y.wc, z.wc), tri_mix(v, x.wc, y.wf, z.wc), tri_mix(w, x.wc, y.wc, z.wf)};
    }
    return Vec3T<T>{far.template at<0>(m.u), far.template at<1>(m.v), far.template at<2>(m.w)};
}

// The displacement of trace_rk2 (ode.h:30-35) or Ralston RK3 (c = 0, 1/2, 3/4; b = 2/9, 1/3, 4/9)
// from the first stage's velocity a; s is the signed step in cells per unit velocity (-dt / dx for
// a backtrace), at(d) the velocity d cells away.
template <typename T, int TRACE, typename F>
__device__ __forceinline__ Vec3T<T> backtrace_from(const Vec3T<T>& a, T s, F&& at) {
    const T s2 = T(0.5) * s;
    const Vec3T<T> b = at(Vec3T<T>{s2 * a.x, s2 * a.y, s2 * a.z});
    if constexpr (TRACE == EL_TRACE_RK2) {
        return Vec3T<T>{s * b.x, s * b.y, s * b.z};
    } else {
        const T s3 = T(0.75) * s;
        const Vec3T<T> c = at(Vec3T<T>{s3 * b.x, s3 * b.y, s3 * b.z});
        const T w1 = s * (T(2) / T(9)), w2 = s * (T(1) / T(3)), w3 = s * (T(4) / T(9));
        return Vec3T<T>{w1 * a.x + w2 * b.x + w3 * c.x, w1 * a.y + w2 * b.y + w3 * c.y,
                        w1 * a.z + w2 * b.z + w3 * c.z};
    }
}

// The velocity at the centre of cell (i, j, k), the first stage of a level-set backtrace: the
// trilinear read there has fractions 1/2 along a component's own axis and 0 along the others,
// so each component is the mean of its two faces (a zero fraction leaves its first value).
// The faces of a cell are inside every grid (no clamping).
template <typename T>
__device__ __forceinline__ Vec3T<T> cell_velocity(const Mac<T>& m, int i, int j, int k) {
    const T* u = m.u.d + cell_index(m.u, i, j, k);
    const T* v = m.v.d + cell_index(m.v, i, j, k);
    const T* w = m.w.d + cell_index(m.w, i, j, k);
    return Vec3T<T>{lerp1(__ldg(u), __ldg(u + 1), T(0.5)), lerp1(__ldg(v), __ldg(v + m.v.n0), T(0.5)),
                    lerp1(__ldg(w), __ldg(w + m.w.n0 * m.w.n1), T(0.5))};
}

// The foot point of cell (i, j, k), as the coordinate among the cells that own_at and sample_weno6
// take after foot_coords: FP64 the displacement, relative to the cell; FP32 the absolute position
// (relative to index 0).  vel(axes, far, stage) reads the velocity of stage 1 or 2.
//
// The FP32 level set is rounded at every operation as it always was: positions are absolute, WENO6
// combines its three candidates, and which product of a lerp is rounded alone (LerpForm) is the
// compiler's choice of one build written down.  The projection is why.  The ghost-fluid fractions
// are ratios of the distances to the surface, so that where a cell lies within 1e-3 dx of it, another
// rounding of phi, a more exact one too, gives another velocity: a cell with phi = -0.00092 dx, phi moved
// by 2e-6 dx, has another pressure by 0.07 %, and its faces' v and w are off by 1e-3 of themselves.  Twelve
// scenes of 0.4 to 2.3 million cells under six seeds, phi from WENO6 relative to its middle
// candidate: twelve fields off by 1e-4 to 1e-3 at single faces (5e-3 under another seed); with
// these roundings no field by 1e-4 under eight.  tests/test_gpu_level_set_bits.py holds the bits.
template <typename T>
__device__ __forceinline__ int foot_base(int i) {
    return sizeof(T) == 4 ? 0 : i;
}
template <int N>
using Stage = std::integral_constant<int, N>;
template <typename T, int TRACE, typename F>
__device__ __forceinline__ Vec3T<T> level_set_foot(const Vec3T<T>& a, int i, int j, int k, T dt, T dx, T inv_dx, F&& vel) {
    if constexpr (sizeof(T) == 8) {
        const Vec3T<T> h{T(0), T(0), T(0)};
        return backtrace_from<T, TRACE>(a, -dt * inv_dx, [&](const Vec3T<T>& d) {
            return vel(axes_rel(i, j, k, h, d), FarRel<T>{i, j, k, h, d}, Stage<1>());
        });
    } else {
        const float h = -dt;
        const Vec3T<float> p{rn_mul(i + 0.5f, dx), rn_mul(j + 0.5f, dx), rn_mul(k + 0.5f, dx)};
        auto step = [](const Vec3T<float>& q, float s, const Vec3T<float>& v) {
            return Vec3T<float>{rn_fma(s, v.x, q.x), rn_fma(s, v.y, q.y), rn_fma(s, v.z, q.z)};
        };
        auto at = [&](const Vec3T<float>& q, auto stage) { return vel(axes_abs(q, dx, inv_dx), FarAbs{q, dx, inv_dx}, stage); };
        const Vec3T<float> b = at(step(p, 0.5f * h, a), Stage<1>());
        Vec3T<float> q;
        if constexpr (TRACE == EL_TRACE_RK2) {
            q = step(p, h, b);
        } else {
            const Vec3T<float> c = at(step(p, 0.75f * h, b), Stage<2>());
            q = step(step(step(p, h * (2.f / 9.f), a), h * (1.f / 3.f), b), h * (4.f / 9.f), c);
        }
        return q;
    }
}

// a coordinate of level_set_foot's point among the cells: FP64 the displacement itself
template <typename T>
__device__ __forceinline__ T foot_coord(T p, T dx, T inv_dx) {
    if constexpr (sizeof(T) == 8)
        return p;
    else
        return rn_mul(rn_sub(p, 0.5f * dx), inv_dx);
}
template <typename T>
__device__ __forceinline__ Vec3T<T> foot_coords(const Vec3T<T>& p, T dx, T inv_dx) {
    return Vec3T<T>{foot_coord(p.x, dx, inv_dx), foot_coord(p.y, dx, inv_dx), foot_coord(p.z, dx, inv_dx)};
}

// out(x) = src(trace(x, -dt)) for every sample of src's grid (comp 0: cell centres, 1..3: a face
// component).
template <typename T, int TRACE, int SAMPLE>
__global__ void __launch_bounds__(256) advect_kernel(GridView<T> src, int comp, T* __restrict__ out, Mac<T> mac,
                                                     DtArg dt, T dx, T inv_dx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= src.n0 || j >= src.n1) return;
    const T dtv = (T)dt_value(dt);
    const Vec3T<T> zero{T(0), T(0), T(0)};
    int bi = i, bj = j, bk = k;
    Vec3T<T> e;
    if (comp == 0) {
        auto vel = [&](const Axes<T>& a, const auto& far, auto) { return velocity_global(mac, a, far); };
        const Vec3T<T> a = velocity_global(mac, axes_rel(i, j, k, zero, zero), FarRel<T>{i, j, k, zero, zero});
        e = foot_coords(level_set_foot<T, TRACE>(a, i, j, k, dtv, dx, inv_dx, vel), dx, inv_dx);
        bi = foot_base<T>(i);
        bj = foot_base<T>(j);
        bk = foot_base<T>(k);
    } else {
        const Vec3T<T> h{comp == 1 ? T(-0.5) : T(0), comp == 2 ? T(-0.5) : T(0), comp == 3 ? T(-0.5) : T(0)};
        auto at = [&](const Vec3T<T>& d) {
            return velocity_global(mac, axes_rel(i, j, k, h, d), FarRel<T>{i, j, k, h, d});
        };
        e = backtrace_from<T, TRACE>(at(zero), -dtv * inv_dx, at);
    }
    T r;
    if constexpr (SAMPLE == EL_SAMPLE_WENO6)
        r = sample_weno6(src, bi, bj, bk, e.x, e.y, e.z);
    else
        r = own_at<T, false>(src, bi, bj, bk, e);
    const int oc = cell_index(src, i, j, k);
    if (EL_IN(oc, (long long)src.n0 * src.n1 * src.n2, 1)) out[oc] = r;
}

// ---------------------------------------------------------------------------------------
// Tiled variants.  Under the CFL limit (cfl <= 1) the foot point and every RK stage lie within
// one cell of the sample, so every trilinear velocity sample of a 32 x 8 x 8 tile of outputs
// reads indices within [tile - 2, tile + 1] of each MAC grid: a CTA stages those boxes of u, v
// and w (40 x 12 x 12 values each) in shared memory once and samples them there.  A sample
// whose 8 points are not all in the box (a larger dt) reads global memory instead, with the
// same arithmetic, so the results do not depend on which path a sample took.  The velocity
// advection computes u, v and w of a tile in one CTA (when the advected field is the advecting
// velocity, as in advect_velocity), sharing the staged boxes; the level set samples phi from
// global memory at the foot point.
//
// The box holds the clamped grid (entry p = value at clamp(box origin + p)), so a sample reads
// its 8 points at the unclamped indices i, i+1 (j, k likewise) with no clamping and gets exactly
// the values of the clamped gather lerp() makes; the 8 reads sit at fixed offsets from one
// address.  Along x a box starts four entries left of the tile (a box copy starts on a 16-byte
// boundary) and holds 40 entries; along y and z the halo is two.
constexpr int kTileX = 32, kTileY = 8, kTileZ = 8, kHalo = 2, kHaloX = 4;
constexpr int kBoxX = kTileX + 2 * kHaloX, kBoxY = kTileY + 2 * kHalo, kBoxZ = kTileZ + 2 * kHalo;
// (Rows 64 words apart in FP32, which leaves no bank conflicts where a floor changes within a warp,
// measured the same in the velocity kernel: 594 against 579 us at 256^3; two CTAs an SM, not three.)
constexpr int kBoxN = kBoxX * kBoxY * kBoxZ;

// trilinear sample from a staged box at box-relative floor indices (x, y, z); false when the 8
// points are not all inside the box.  CHECK = false: the caller knows they are (see
// advect_velocity_tiled_kernel)
template <typename T, bool CHECK, int ZF = LERP_ANY>
__device__ __forceinline__ bool staged_lerp(const T* box, int x, int y, int z, T fx, T fy, T fz, T& out) {
    if (CHECK && ((unsigned)x >= (unsigned)(kBoxX - 1) || (unsigned)y >= (unsigned)(kBoxY - 1) ||
                  (unsigned)z >= (unsigned)(kBoxZ - 1)))
        return false;
    const T* p = box + (z * kBoxY + y) * kBoxX + x;
    constexpr int SY = kBoxX, SZ = kBoxX * kBoxY;
    out = tri_mix<T, ZF>(fx, fy, fz, p[0], p[1], p[SY], p[SY + 1], p[SZ], p[SZ + 1], p[SZ + SY], p[SZ + SY + 1]);
    return true;
}

template <typename T>
struct StagedMac {
    const T* box;         // shared memory: the boxes of u, v, w, each [z][y][x]
    int bx0, by0, bz0;    // grid index of the boxes' first entry
};

// u, v, w at one position through the staged boxes; ZU, ZV, ZW: the forms of their z lerps
template <typename T, bool CHECK, int ZU = LERP_ANY, int ZV = LERP_ANY, int ZW = LERP_ANY, typename FAR>
__device__ __forceinline__ Vec3T<T> velocity_staged(const Mac<T>& m, const StagedMac<T>& b, const Axes<T>& a,
                                                    const FAR& far) {
    auto rel = [](int g, int b0) { return (int)((unsigned)g - (unsigned)b0); };
    const AxisCF<T>&x = a.x, &y = a.y, &z = a.z;
    const int xc = rel(x.c, b.bx0), xf = rel(x.f, b.bx0), yc = rel(y.c, b.by0), yf = rel(y.f, b.by0);
    const int zc = rel(z.c, b.bz0), zf = rel(z.f, b.bz0);
    Vec3T<T> v;
    if (!staged_lerp<T, CHECK, ZU>(b.box, xf, yc, zc, x.wf, y.wc, z.wc, v.x) && CHECK) v.x = far.template at<0>(m.u);
    if (!staged_lerp<T, CHECK, ZV>(b.box + kBoxN, xc, yf, zc, x.wc, y.wf, z.wc, v.y) && CHECK) v.y = far.template at<1>(m.v);
    if (!staged_lerp<T, CHECK, ZW>(b.box + 2 * kBoxN, xc, yc, zf, x.wc, y.wc, z.wf, v.z) && CHECK)
        v.z = far.template at<2>(m.w);
    return v;
}

// The velocity at the centre of a face of component C, the first stage of its backtrace: the
// trilinear read there has fractions 0 and 1/2 only, so it is the face's own value and the
// four-point means of the two other components, in the trilinear read's order (x, then y, then
// z; a zero fraction leaves its first value).  (I, J, K): the face, relative to the boxes.  Every
// point lies in the staged boxes (their halos are at least one entry), which hold the clamped grid.
template <typename T>
__device__ __forceinline__ T mid4(T a, T b, T c, T d) {
    return lerp1(lerp1(a, b, T(0.5)), lerp1(c, d, T(0.5)), T(0.5));
}

// pairs of two samples' values: each lane rounded as the scalar operation
__device__ __forceinline__ float2 operator*(float s, float2 v) { return __fmul2_rn(make_float2(s, s), v); }
__device__ __forceinline__ float2 lerp1(float2 a, float2 b, float2 f) {
    const float2 g = __ffma2_rn(f, make_float2(-1.f, -1.f), make_float2(1.f, 1.f));  // 1 - f, one rounding
    return __ffma2_rn(f, b, __fmul2_rn(g, a));
}
__device__ __forceinline__ float2 lerp1(float2 a, float2 b, float f) { return lerp1(a, b, make_float2(f, f)); }
__device__ __forceinline__ float2 mid4(float2 a, float2 b, float2 c, float2 d) {
    return lerp1(lerp1(a, b, 0.5f), lerp1(c, d, 0.5f), 0.5f);
}

// box entries around the face: M(component, di, dj, dk)
template <typename V, int C, typename F>
__device__ __forceinline__ Vec3T<V> face_velocity(F&& M) {
    if constexpr (C == 0)
        return Vec3T<V>{M(0, 0, 0, 0), mid4(M(1, -1, 0, 0), M(1, 0, 0, 0), M(1, -1, 1, 0), M(1, 0, 1, 0)),
                        mid4(M(2, -1, 0, 0), M(2, 0, 0, 0), M(2, -1, 0, 1), M(2, 0, 0, 1))};
    else if constexpr (C == 1)
        return Vec3T<V>{mid4(M(0, 0, -1, 0), M(0, 1, -1, 0), M(0, 0, 0, 0), M(0, 1, 0, 0)), M(1, 0, 0, 0),
                        mid4(M(2, 0, -1, 0), M(2, 0, 0, 0), M(2, 0, -1, 1), M(2, 0, 0, 1))};
    else
        return Vec3T<V>{mid4(M(0, 0, 0, -1), M(0, 1, 0, -1), M(0, 0, 0, 0), M(0, 1, 0, 0)),
                        mid4(M(1, 0, 0, -1), M(1, 0, 1, -1), M(1, 0, 0, 0), M(1, 0, 1, 0)), M(2, 0, 0, 0)};
}

// The largest |value| met, NaN once one was met.  FP32: a three-input maximum of magnitudes that
// keeps NaN; FP64: the high word of the magnitude on the integer pipe (NaN's is above every
// number's), read back as a bound from above.
template <typename T>
struct AbsMax;
template <>
struct AbsMax<float> {
    float m = 0.f;
    __device__ __forceinline__ void add(float a, float b) {
        asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(m), "f"(a), "f"(b));
    }
    __device__ __forceinline__ void add16(const float* p) {
        const float4 q = *reinterpret_cast<const float4*>(p);
        add(q.x, q.y);
        add(q.z, q.w);
    }
    __device__ __forceinline__ void add(float a) { add(a, a); }
    __device__ __forceinline__ AbsMax shuffled(int o) const { return AbsMax{__shfl_xor_sync(0xffffffffu, m, o)}; }
    __device__ __forceinline__ void join(const AbsMax& o) { add(o.m, o.m); }
    __device__ __forceinline__ float value() const { return m; }
};
template <>
struct AbsMax<double> {
    unsigned m = 0;
    __device__ __forceinline__ void add(double a) { m = max(m, (unsigned)__double2hiint(a) & 0x7fffffffu); }
    __device__ __forceinline__ void add16(const double* p) {
        const double2 q = *reinterpret_cast<const double2*>(p);
        add(q.x);
        add(q.y);
    }
    __device__ __forceinline__ AbsMax shuffled(int o) const { return AbsMax{__shfl_xor_sync(0xffffffffu, m, o)}; }
    __device__ __forceinline__ void join(const AbsMax& o) { m = max(m, o.m); }
    __device__ __forceinline__ double value() const { return __hiloint2double((int)m, -1); }
};

// A box that arrived by a box copy (rows of PITCH entries, of which the first BX are used), made
// the clamped box: an entry outside the grid takes the value of its clamped entry (inside the
// grid, so the copy filled it), one warp per row; with MAX, vmax gathers the largest |value| of the
// entries inside the grid (the values the clamped box holds).  A box that lies inside the grid is
// only scanned for vmax, in 16-byte reads.
template <typename T, int BX, int BY, int BZ, bool MAX, int PITCH = BX>
__device__ __forceinline__ void finish_box(T* box, const GridView<T>& g, int bx0, int by0, int bz0, AbsMax<T>& vmax) {
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nthr = blockDim.x * blockDim.y * blockDim.z;
    const bool edge = bx0 < 0 || by0 < 0 || bz0 < 0 || bx0 + BX > g.n0 || by0 + BY > g.n1 || bz0 + BZ > g.n2;
    if (!edge) {
        if constexpr (MAX) {
            constexpr int per = 16 / (int)sizeof(T), row = BX / per;
            static_assert(BX % per == 0 && PITCH % per == 0, "whole 16-byte reads");
#pragma unroll 4
            for (int e = tid; e < row * BY * BZ; e += nthr) vmax.add16(box + (e / row) * PITCH + (e % row) * per);
        }
        return;
    }
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    for (int row = warp; row < BY * BZ; row += nwarps) {
        const int bz = row / BY, by = row - bz * BY;
        const int cy = clampi(by0 + by, 0, g.n1 - 1) - by0, cz = clampi(bz0 + bz, 0, g.n2 - 1) - bz0;
        const bool row_in = cy == by && cz == bz;
        const T* src = box + (cz * BY + cy) * PITCH;
        T* dst = box + row * PITCH;
        for (int x = lane; x < BX; x += 32) {
            const int cx = clampi(bx0 + x, 0, g.n0 - 1) - bx0;
            if (row_in && cx == x) {
                if (MAX) vmax.add(dst[x]);
            } else {
                dst[x] = src[cx];
            }
        }
    }
}

// Issues the box copies of a tile (one thread; the mbarrier is the CTA's own), `bytes` in all.
__device__ __forceinline__ void copy_boxes_begin(uint64_t* bar, unsigned bytes) {
    mbar_init(bar, 1);
    mbar_init_fence();
    mbar_expect_tx(bar, bytes);
}

// Every thread waits (bounded) for the CTA's box copies; true, the same in every thread, when a
// wait gave up.  Then the fault is recorded and one thread waits once more (bounded) so that no
// copy is still landing when the CTA ends.  Call after a barrier that follows the mbarrier's
// initialisation.
__device__ __forceinline__ bool copy_boxes_failed(uint64_t* bar, bool report) {
    const bool ok = mbar_wait(bar, 0);
    if (!__syncthreads_or(!ok)) return false;
    if (threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0) {
        if (report) atomicOr(&advect_wait_fault, 1u);
        mbar_wait(bar, 0);
    }
    __syncthreads();
    return true;
}

// NaN into a thread's outputs of a tile whose boxes did not arrive (rows j, planes z0 .. z0+nz-1)
template <typename T>
__device__ __forceinline__ void nan_column(const GridView<T>& g, T* __restrict__ o, int i, int j, int z0, int nz) {
    if (i >= g.n0 || j >= g.n1) return;
    for (int kk = 0; kk < nz && z0 + kk < g.n2; ++kk) {
        const int oc = cell_index(g, i, j, z0 + kk);
        if (EL_IN(oc, (long long)g.n0 * g.n1 * g.n2, 4)) o[oc] = std::numeric_limits<T>::quiet_NaN();
    }
}

// Stages the clamped boxes of u, v, w around tile (x0, y0, z0): a component with a box map by a
// box copy (then finish_box), the others by plain loads (the first 32 entries of a row one warp a
// row, the last 8 of all rows by all threads).  vmax gathers the largest |value| this thread staged
// or scanned (NaN if it met one).  `failed`: the box copies did not arrive (the same in every
// thread).
template <typename T>
__device__ __forceinline__ void stage_plain(const GridView<T>& g, T* box, int bx0, int by0, int bz0, int tid, int nthr,
                                            AbsMax<T>& vmax) {
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    auto row_of = [&](int row) {
        const int bz = row / kBoxY, by = row - bz * kBoxY;
        const int gy = clampi(by0 + by, 0, g.n1 - 1), gz = clampi(bz0 + bz, 0, g.n2 - 1);
        return g.d + (long long)g.n0 * (gy + (long long)g.n1 * gz);
    };
    const int gx = clampi(bx0 + lane, 0, g.n0 - 1);
#pragma unroll 6
    for (int row = warp; row < kBoxY * kBoxZ; row += nwarps) {
        const T v = __ldg(row_of(row) + gx);
        box[row * kBoxX + lane] = v;
        vmax.add(v);
    }
    constexpr int kTail = kBoxX - 32;
    const int tx = clampi(bx0 + 32 + tid % kTail, 0, g.n0 - 1);
#pragma unroll 2
    for (int e = tid; e < kTail * kBoxY * kBoxZ; e += nthr) {
        const T v = __ldg(row_of(e / kTail) + tx);
        box[(e / kTail) * kBoxX + 32 + tid % kTail] = v;
        vmax.add(v);
    }
}

template <typename T>
__device__ __forceinline__ StagedMac<T> stage_mac(const Mac<T>& m, const MacMaps& maps, T* smem, uint64_t* bar,
                                                  int x0, int y0, int z0, AbsMax<T>& vmax, bool& failed) {
    const int bx0 = x0 - kHaloX, by0 = y0 - kHalo, bz0 = z0 - kHalo;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y, nthr = blockDim.x * blockDim.y;
    // the flags in registers (a parameter indexed at run time would be copied to local memory)
    const bool on0 = maps.c[0].on != 0, on1 = maps.c[1].on != 0, on2 = maps.c[2].on != 0;
    const int ncopy = (int)on0 + (int)on1 + (int)on2;
    if (ncopy && tid == 0) {
        copy_boxes_begin(bar, (unsigned)(ncopy * kBoxN * sizeof(T)));
        if (on0) tma_load_3d(smem, &maps.c[0].m, bar, bx0, by0, bz0);
        if (on1) tma_load_3d(smem + kBoxN, &maps.c[1].m, bar, bx0, by0, bz0);
        if (on2) tma_load_3d(smem + 2 * kBoxN, &maps.c[2].m, bar, bx0, by0, bz0);
    }
    if (!on0) stage_plain(m.u, smem, bx0, by0, bz0, tid, nthr, vmax);
    if (!on1) stage_plain(m.v, smem + kBoxN, bx0, by0, bz0, tid, nthr, vmax);
    if (!on2) stage_plain(m.w, smem + 2 * kBoxN, bx0, by0, bz0, tid, nthr, vmax);
    failed = false;
    if (ncopy) {
        __syncthreads();  // the mbarrier's initialisation is seen by every thread
        failed = copy_boxes_failed(bar, maps.c[0].on == BOX_REPORTED || maps.c[1].on == BOX_REPORTED ||
                                            maps.c[2].on == BOX_REPORTED);
        if (!failed) {
            if (on0) finish_box<T, kBoxX, kBoxY, kBoxZ, true>(smem, m.u, bx0, by0, bz0, vmax);
            if (on1) finish_box<T, kBoxX, kBoxY, kBoxZ, true>(smem + kBoxN, m.v, bx0, by0, bz0, vmax);
            if (on2) finish_box<T, kBoxX, kBoxY, kBoxZ, true>(smem + 2 * kBoxN, m.w, bx0, by0, bz0, vmax);
        }
    }
    return StagedMac<T>{smem, bx0, by0, bz0};
}

// The largest |velocity| the CTA staged (NaN if it staged a NaN; FP64: a bound from above), as the
// same value in every thread.  Call after the staging, in place of the __syncthreads that ends it.
template <typename T>
__device__ __forceinline__ T box_max(AbsMax<T> vmax) {
    __shared__ decltype(vmax.m) wmax[kTileX * kTileY / 32];
    for (int o = 16; o > 0; o >>= 1) vmax.join(vmax.shuffled(o));
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    if ((tid & 31) == 0) wmax[tid >> 5] = vmax.m;
    __syncthreads();
    AbsMax<T> m;
#pragma unroll
    for (int q = 0; q < kTileX * kTileY / 32; ++q) m.join(AbsMax<T>{wmax[q]});
    return m.value();
}

// A step moves no sample more than one cell when |v| |dt| / dx < 1 over the staged boxes (every
// RK stage and the foot point are convex combinations of velocities read inside the boxes, by
// induction): then all of a tile's staged reads fall inside its boxes (the halo is two cells)
// and the reads need no check.  False for a NaN or infinite velocity or dt.
// s: the step in cells per unit velocity
template <typename T>
__device__ __forceinline__ bool within_one_cell(T vmax, T s) {
    const T reach = vmax * (s < T(0) ? -s : s);
    return reach <= T(0.999);
}

// one sample of component C (CHECK: each staged read is checked and falls back to the global read
// outside the box)
template <typename T, int TRACE, bool CHECK, int C>
__device__ __forceinline__ void velocity_sample(const Mac<T>& mac, const GridView<T>& g, const StagedMac<T>& sm,
                                                T* __restrict__ o, T s, int i, int j, int k) {
    if (i >= g.n0 || j >= g.n1 || k >= g.n2) return;
    const T* own = sm.box + C * kBoxN;
    const int I = i - sm.bx0, J = j - sm.by0, K = k - sm.bz0;
    const Vec3T<T> h{C == 0 ? T(-0.5) : T(0), C == 1 ? T(-0.5) : T(0), C == 2 ? T(-0.5) : T(0)};
    const Vec3T<T> a = face_velocity<T, C>([&](int c, int di, int dj, int dk) {
        return sm.box[c * kBoxN + ((K + dk) * kBoxY + J + dj) * kBoxX + I + di];
    });
    const Vec3T<T> d = backtrace_from<T, TRACE>(a, s, [&](const Vec3T<T>& e) {
        return velocity_staged<T, CHECK, LERP_A, LERP_A, LERP_A>(mac, sm, axes_rel(i, j, k, h, e), FarRel<T>{i, j, k, h, e});
    });
    int x, y, z;
    T fx, fy, fz, r;
    floor_index(d.x, x, fx);
    floor_index(d.y, y, fy);
    floor_index(d.z, z, fz);
    if (!staged_lerp<T, CHECK, LERP_A>(own, (int)((unsigned)I + (unsigned)x), (int)((unsigned)J + (unsigned)y),
                               (int)((unsigned)K + (unsigned)z), fx, fy, fz, r) &&
        CHECK)
        r = tri_clamped(g, i, j, k, d.x, d.y, d.z);
    const int oc = cell_index(g, i, j, k);
    if (EL_IN(oc, (long long)g.n0 * g.n1 * g.n2, 2)) o[oc] = r;
}

// Two samples of component C, (i, j, k) and (i, j, k + 1), in packed float2 arithmetic from the
// boxes to the result: every quantity is a pair of the two samples' values, so no lanes are moved
// between pairs (with the halves of one trilinear read as the pair, a third of the instructions
// moved registers).  Each lane is rounded as velocity_sample's scalars.  Only for tiles in which
// every read lies in the boxes.
// a pair of floors as byte offsets (times `stride`, plus `base`), and the fractions
struct AxisPair {
    unsigned a, b;
    float2 w;
};
__device__ __forceinline__ AxisPair axis_pair(float2 e, unsigned base, unsigned stride) {
    const float big = 12582912.0f;  // as floor_index
    const float2 r = __fadd2_rd(e, make_float2(big, big));
    const float2 fl = __fadd2_rn(r, make_float2(-big, -big));
    AxisPair p;
    p.w = __ffma2_rn(fl, make_float2(-1.f, -1.f), e);  // e - fl (packed additions take no negated operand)
    // the magic number's bits fold into the base (unsigned arithmetic wraps)
    const unsigned c = base - 0x4B400000u * stride;
    // as instructions: with the product written in C++, nvcc 13.0.88 folded it into an address without
    // the stride (found by the index check of tri_pair in the debug build; not reduced to a small case)
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(p.a) : "r"(__float_as_int(r.x)), "r"(stride), "r"(c));
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(p.b) : "r"(__float_as_int(r.y)), "r"(stride), "r"(c));
    return p;
}

// byte strides of a box
constexpr unsigned kSX = 4, kSY = 4 * kBoxX, kSZ = kSY * kBoxY;

// the entry at shared-memory byte address `at` + OFF (the clobber keeps it behind the barrier that ends
// the staging)
template <int OFF>
__device__ __forceinline__ float lds(unsigned at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1 + %2];" : "=f"(v) : "r"(at), "n"(OFF) : "memory");
    return v;
}

// trilinear reads of a pair of samples, the second one plane above, from the box at byte offset BOX
// (box0: the boxes' shared-memory address)
template <int BOX>
__device__ __forceinline__ float2 tri_pair(unsigned box0, const AxisPair& x, const AxisPair& y, const AxisPair& z) {
    unsigned p = x.a + y.a + z.a, q = x.b + y.b + z.b;
    constexpr int SX = kSX, SY = kSY, SZ = kSZ, UP = BOX + SZ;
    if (!EL_IN(p - box0, 4 * kBoxN - SX - SY - SZ, 5) || !EL_IN(q - box0, 4 * kBoxN - SX - SY - 2 * SZ, 6)) p = q = box0;
    // Every read is in the box, see the callers.  An address that was not would read the box's end instead
    // of faulting; the debug build records it (above).
    p = box0 + min(p - box0, (unsigned)(4 * kBoxN - SX - SY - SZ - 4));
    q = box0 + min(q - box0, (unsigned)(4 * kBoxN - SX - SY - 2 * SZ - 4));
    const float2 x00 = lerp1(make_float2(lds<BOX>(p), lds<UP>(q)), make_float2(lds<BOX + SX>(p), lds<UP + SX>(q)), x.w);
    const float2 x10 = lerp1(make_float2(lds<BOX + SY>(p), lds<UP + SY>(q)),
                             make_float2(lds<BOX + SY + SX>(p), lds<UP + SY + SX>(q)), x.w);
    const float2 x01 = lerp1(make_float2(lds<BOX + SZ>(p), lds<UP + SZ>(q)),
                             make_float2(lds<BOX + SZ + SX>(p), lds<UP + SZ + SX>(q)), x.w);
    const float2 x11 = lerp1(make_float2(lds<BOX + SZ + SY>(p), lds<UP + SZ + SY>(q)),
                             make_float2(lds<BOX + SZ + SY + SX>(p), lds<UP + SZ + SY + SX>(q)), x.w);
    return lerp1(lerp1(x00, x10, y.w), lerp1(x01, x11, y.w), z.w);
}

template <int TRACE, int C>
__device__ __forceinline__ void velocity_pair(const GridView<float>& g, const StagedMac<float>& sm,
                                              float* __restrict__ o, float s, int i, int j, int k) {
    if (i >= g.n0 || j >= g.n1 || k >= g.n2) return;
    const unsigned box0 = (unsigned)__cvta_generic_to_shared(sm.box);
    const unsigned I = kSX * (i - sm.bx0) + box0;
    const unsigned J = kSY * (j - sm.by0), K = kSZ * (k - sm.bz0);
    constexpr int B = 4 * kBoxN;  // bytes of a box
    constexpr int P = kBoxX;
    const float* centre = sm.box + ((k - sm.bz0) * kBoxY + j - sm.by0) * P + i - sm.bx0;
    const Vec3T<float2> a = face_velocity<float2, C>([&](int c, int di, int dj, int dk) {
        const float* p = centre + (c * kBoxN + (dk * kBoxY + dj) * P + di);
        return make_float2(p[0], p[P * kBoxY]);
    });
    auto cell = [](float2 d, bool face_axis) { return face_axis ? __fadd2_rn(d, make_float2(-0.5f, -0.5f)) : d; };
    auto face = [](float2 d, bool face_axis) { return face_axis ? d : __fadd2_rn(d, make_float2(0.5f, 0.5f)); };
    auto at = [&](float2 dx, float2 dy, float2 dz) {
        const AxisPair xc = axis_pair(cell(dx, C == 0), I, kSX), xf = axis_pair(face(dx, C == 0), I, kSX);
        const AxisPair yc = axis_pair(cell(dy, C == 1), J, kSY), yf = axis_pair(face(dy, C == 1), J, kSY);
        const AxisPair zc = axis_pair(cell(dz, C == 2), K, kSZ), zf = axis_pair(face(dz, C == 2), K, kSZ);
        return Vec3T<float2>{tri_pair<0>(box0, xf, yc, zc), tri_pair<B>(box0, xc, yf, zc), tri_pair<2 * B>(box0, xc, yc, zf)};
    };
    const float s2 = 0.5f * s;
    const Vec3T<float2> b = at(s2 * a.x, s2 * a.y, s2 * a.z);
    Vec3T<float2> d;
    if constexpr (TRACE == EL_TRACE_RK2) {
        d = Vec3T<float2>{s * b.x, s * b.y, s * b.z};
    } else {
        const float s3 = 0.75f * s;
        const Vec3T<float2> c = at(s3 * b.x, s3 * b.y, s3 * b.z);
        const float w1 = s * (2.f / 9.f), w2 = s * (1.f / 3.f), w3 = s * (4.f / 9.f);
        auto sum = [&](float2 p, float2 q, float2 r) {
            return __ffma2_rn(make_float2(w3, w3), r, __ffma2_rn(make_float2(w2, w2), q, w1 * p));
        };
        d = Vec3T<float2>{sum(a.x, b.x, c.x), sum(a.y, b.y, c.y), sum(a.z, b.z, c.z)};
    }
    const float2 r = tri_pair<C * B>(box0, axis_pair(d.x, I, kSX), axis_pair(d.y, J, kSY), axis_pair(d.z, K, kSZ));
    const int oc = cell_index(g, i, j, k), plane = g.n0 * g.n1;
    if (EL_IN(oc, (long long)plane * g.n2, 2)) o[oc] = r.x;
    if (k + 1 < g.n2 && EL_IN(oc + plane, (long long)plane * g.n2, 2)) o[oc + plane] = r.y;
}

// The u, v, w samples of a tile of cells.  A component has one more sample than cells along its own
// axis: where the last tile is full, it also takes that column, row or plane of faces (one entry
// beyond the tile, which the boxes' halos serve along that axis) rather than a further tile
// staging three boxes for them.
template <typename T, int TRACE, bool CHECK>
__device__ __forceinline__ void velocity_tile(const Mac<T>& mac, const StagedMac<T>& sm, T* __restrict__ ou,
                                              T* __restrict__ ov, T* __restrict__ ow, T s, int x0, int y0, int z0) {
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i = x0 + tx, j = y0 + ty;
    const bool more_u = x0 + kTileX == mac.u.n0 - 1, more_v = y0 + kTileY == mac.v.n1 - 1;
    const bool more_w = z0 + kTileZ == mac.w.n2 - 1;
    if constexpr (sizeof(T) == 4 && !CHECK) {
#pragma unroll 1
        for (int kk = 0; kk < kTileZ; kk += 2) {
            velocity_pair<TRACE, 0>(mac.u, sm, ou, s, i, j, z0 + kk);
            velocity_pair<TRACE, 1>(mac.v, sm, ov, s, i, j, z0 + kk);
            velocity_pair<TRACE, 2>(mac.w, sm, ow, s, i, j, z0 + kk);
        }
    } else {
#pragma unroll 1
        for (int kk = 0; kk < kTileZ; ++kk) {
            velocity_sample<T, TRACE, CHECK, 0>(mac, mac.u, sm, ou, s, i, j, z0 + kk);
            velocity_sample<T, TRACE, CHECK, 1>(mac, mac.v, sm, ov, s, i, j, z0 + kk);
            velocity_sample<T, TRACE, CHECK, 2>(mac, mac.w, sm, ow, s, i, j, z0 + kk);
        }
    }
    // 8 x 8 faces by two warps, 32 x 8 by all
    if (more_u && ty < 2) velocity_sample<T, TRACE, CHECK, 0>(mac, mac.u, sm, ou, s, x0 + kTileX, y0 + (tx & 7), z0 + 4 * ty + (tx >> 3));
    if (more_v) velocity_sample<T, TRACE, CHECK, 1>(mac, mac.v, sm, ov, s, i, y0 + kTileY, z0 + ty);
    if (more_w) velocity_sample<T, TRACE, CHECK, 2>(mac, mac.w, sm, ow, s, i, j, z0 + kTileZ);
}

// u, v, w of a tile, each advected through the (old) velocity itself.  FP32: bound by shared-memory
// loads (66 a sample, seven trilinear reads) and issue (285 instructions a sample, from 617):
// 256^3 RK3 0.96 -> 0.58 ms, three per-sample launches of 256 x 128 x 192 took 0.62 ms for what
// now takes 0.24.  FP64: bound by its FP64 operations (350 a sample before, now half of that): 128^3 RK3 5.04 ->
// 2.03 ms.
template <typename T, int TRACE>
__global__ void __launch_bounds__(kTileX * kTileY, sizeof(T) == 4 ? 3 : 1) advect_velocity_tiled_kernel(
    Mac<T> mac, T* __restrict__ ou, T* __restrict__ ov, T* __restrict__ ow, DtArg dt, T inv_dx,
    const __grid_constant__ MacMaps maps) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* smem = reinterpret_cast<T*>(align128(smem_raw));
    __shared__ uint64_t bar;
    const int x0 = blockIdx.x * kTileX, y0 = blockIdx.y * kTileY, z0 = blockIdx.z * kTileZ;
    AbsMax<T> vmax;
    bool failed;
    const StagedMac<T> sm = stage_mac(mac, maps, smem, &bar, x0, y0, z0, vmax, failed);
    if (failed) {
        const int i = x0 + threadIdx.x, j = y0 + threadIdx.y;
        // the samples velocity_tile would have written: the tile's, and the last faces of a last tile
        const bool more_w = z0 + kTileZ == mac.w.n2 - 1;
        nan_column(mac.u, ou, i, j, z0, kTileZ);
        nan_column(mac.v, ov, i, j, z0, kTileZ);
        nan_column(mac.w, ow, i, j, z0, kTileZ + (more_w ? 1 : 0));
        if (threadIdx.x == 0 && x0 + kTileX == mac.u.n0 - 1) nan_column(mac.u, ou, x0 + kTileX, j, z0, kTileZ);
        if (threadIdx.y == 0 && y0 + kTileY == mac.v.n1 - 1) nan_column(mac.v, ov, i, y0 + kTileY, z0, kTileZ);
        return;
    }
    const T bm = box_max(vmax);  // ends the staging (a barrier)
    const T s = -(T)dt_value(dt) * inv_dx;
    if (within_one_cell(bm, s))
        velocity_tile<T, TRACE, false>(mac, sm, ou, ov, ow, s, x0, y0, z0);
    else
        velocity_tile<T, TRACE, true>(mac, sm, ou, ov, ow, s, x0, y0, z0);
}

// the level set (cells) through the staged velocity; phi itself from global memory (trilinear)
template <typename T, int TRACE>
__global__ void __launch_bounds__(kTileX * kTileY) advect_phi_tiled_kernel(GridView<T> src, T* __restrict__ out,
                                                                           Mac<T> mac, DtArg dt, T dx, T inv_dx,
                                                                           const __grid_constant__ MacMaps maps) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* smem = reinterpret_cast<T*>(align128(smem_raw));
    __shared__ uint64_t bar;
    const int x0 = blockIdx.x * kTileX, y0 = blockIdx.y * kTileY, z0 = blockIdx.z * kTileZ;
    AbsMax<T> vmax;
    bool failed;
    const StagedMac<T> sm = stage_mac(mac, maps, smem, &bar, x0, y0, z0, vmax, failed);
    if (failed) {
        nan_column(src, out, x0 + threadIdx.x, y0 + threadIdx.y, z0, kTileZ);
        return;
    }
    const T dtv = (T)dt_value(dt);
    const bool inside = within_one_cell(box_max(vmax), dtv * inv_dx);  // ends the staging
    const int i = x0 + threadIdx.x, j = y0 + threadIdx.y;
    if (i >= src.n0 || j >= src.n1) return;
#pragma unroll 1
    for (int kk = 0; kk < kTileZ; ++kk) {
        const int k = z0 + kk;
        if (k >= src.n2) break;
        const Vec3T<T> a = cell_velocity(mac, i, j, k);
        Vec3T<T> e;
        if (inside)
            e = level_set_foot<T, TRACE>(a, i, j, k, dtv, dx, inv_dx, [&](const Axes<T>& q, const auto& far, auto stage) {
                constexpr int N = decltype(stage)::value;
                constexpr int UV = N == 2 ? LERP_A : LERP_B, W = TRACE == EL_TRACE_RK2 ? LERP_A : LERP_B;
                return velocity_staged<T, false, UV, UV, W>(mac, sm, q, far);
            });
        else
            e = level_set_foot<T, TRACE>(a, i, j, k, dtv, dx, inv_dx, [&](const Axes<T>& q, const auto& far, auto) {
                return velocity_staged<T, true>(mac, sm, q, far);
            });
        const int oc = cell_index(src, i, j, k);
        const T r = own_at<T, true>(src, foot_base<T>(i), foot_base<T>(j), foot_base<T>(k), foot_coords(e, dx, inv_dx));
        if (EL_IN(oc, (long long)src.n0 * src.n1 * src.n2, 3)) out[oc] = r;
    }
}

// ---------------------------------------------------------------------------------------
// WENO6 level set, tiled.  Under the CFL limit the foot point of a cell lies within one cell
// of it, so the 6^3 stencils of a 32 x 8 x WZ tile of cells read phi within [tile - 3, tile + 4]:
// the CTA stages that clamped box (39 x 15 x (WZ + 7) nodes) once, by one box copy where the cell
// grid's row pitch allows it (along x it then starts four cells left of the tile, a 16-byte
// boundary, and holds 40 entries, of which the first is never read).
//
// The smoothness indicators of an x-pass depend only on the six values it reads, not on the
// sample's fraction, so they are formed once per (row, floor index) of the box (34 floor indices of
// each row) and shared by every sample whose stencil uses that row segment, instead of being formed
// by each of the 36 x-passes of every sample.  The y- and z-passes combine per-sample values and are
// evaluated in full.
//
// FP32: an entry is the three reciprocal squares (weno6_sq2) in 16 bytes; the expressions are those of
// weno6_sq2, weno6_combine2 and, for the z-pass, weno6_eval, so that every sample within a cell of
// its four planes has the same bits whatever the tile (level_set_foot says why).  Bound by
// instruction issue; 256^3 1.43 ms (1.07 with the FP64 form below in float, which the bits rule out).
//
// FP64: the six-point combination relative to its middle candidate.  Neighbouring candidates are cubics
// through three common nodes, so they differ by a fourth difference times a fixed polynomial:
//   p_a - p_b = -D0 (x+1) x (x-1) / 6,   p_c - p_b = D1 x (x-1) (x-2) / 6,
//   D0 = v4 - 4 v3 + 6 v2 - 4 v1 + v0,   D1 = v5 - 4 v4 + 6 v3 - 4 v2 + v1,
// and with the nonlinear weights alpha_s = C_s / q_s, q_s = (eps + IS_s)^2, taken relative to the
// middle one (ra = qb / qa, rc = qb / qc),
//   sum(alpha p) / sum(alpha) = p_b + (Ka ra D0 + Kc rc D1) / (Cb + Ca ra + Cc rc),
// Ka = -Ca (x+1) x (x-1) / 6, Kc = Cc x (x-1) (x-2) / 6: one candidate instead of three, and one
// division instead of four.  An entry is {ra, rc} and the plane of D0 (D1 is the next floor index's
// D0), three doubles.  Bound by the FP64 operations (1400 a sample; 128^3: 11.2 -> 5.6 ms).
//
// A foot point outside the box (a larger dt), and in FP64 a result that is not finite, takes the
// global sample_weno6 path: its weights alpha_s stay finite where ratios of the q_s overflow.
constexpr int kWX = 32, kWY = 8;
constexpr int kWNodes = kWX + 8, kWBY = kWY + 7;  // nodes [tile - 4, tile + 4] x [tile - 3, tile + 4]
constexpr int kWBases = kWX + 2;               // floor indices [tile - 1, tile + 32]

template <typename T, int WZ, int NZ>
struct WenoTile {
    static constexpr int kBZ = WZ + 7;             // nodes [tile - 3, tile + 4] along z
    static constexpr int kRows = kWBY * kBZ;
    // FP32: rows of the box and of the entries a multiple of 32 banks apart, so that lanes whose
    // foot points lie in neighbouring rows do not meet on a bank
    static constexpr int kBX = sizeof(T) == 4 ? 64 : kWNodes;
    static constexpr int kEP = sizeof(T) == 4 ? 40 : kWBases;
    static constexpr int kBoxN = kBX * kRows;      // phi box (a multiple of 16 bytes)
    static constexpr int kEntries = kRows * kWBases;
    static constexpr int kDiffs = kWBases + 1;     // FP64: D0 of the floor indices and of one more
    static constexpr int kFoot = kWX * kWY * WZ;   // FP32: the samples' foot points, x, y, z planes
    static constexpr int kBytes =
        kBoxN * (int)sizeof(T) + kRows * kEP * 16 + (sizeof(T) == 4 ? kFoot * 12 : kRows * kDiffs * 8);
    static constexpr int kNZ = NZ;                 // planes at a time
    static constexpr int kThreads = kWX * kWY * kNZ;
};

// the part of the FP64 combination that depends on x only
struct WenoX {
    double L[4];  // p_b = sum_m L[m] v[m + 1]
    double Ca, Cb, Cc, Ka, Kc;
};

__device__ __forceinline__ WenoX weno_x(double x) {
    WenoX w;
    const double xp = x + 1.0, xm = x - 1.0, x2 = x - 2.0;
    // p_b in Newton form on nodes -1, 0, 1, 2
    const double n2 = xp * x * 0.5, n3 = xp * x * xm * (1.0 / 6.0);
    w.L[0] = 1.0 - xp + n2 - n3;
    w.L[1] = xp - 2.0 * n2 + 3.0 * n3;
    w.L[2] = n2 - 3.0 * n3;
    w.L[3] = n3;
    w.Ca = (2.0 - x) * (3.0 - x) * (1.0 / 20.0);
    w.Cb = (3.0 - x) * (x + 2.0) * (1.0 / 10.0);
    w.Cc = (x + 2.0) * xp * (1.0 / 20.0);
    w.Ka = -w.Ca * n3;
    w.Kc = w.Cc * (x * xm * x2 * (1.0 / 6.0));
    return w;
}

// q_s = (eps + IS_s)^2 of the three candidates, times a common factor, and the fourth differences
// D0, D1.  Each 180 IS_s is 244 times a sum of squares of combinations of the first differences
// (the quadratic form factored from its leading term; IS_2's is IS_0's read from the right):
//   form(a, b, c) = (a + B b + G c)^2 + D (b + E c)^2 + Z c^2,
// nine operations with the square.  The common factor (244 / 180)^2 drops out of the weights' ratios
// and, with eps scaled alike, out of their normalisation.
__device__ __forceinline__ void weno_q(const double (&v)[6], double& qa, double& qb, double& qc, double& D0,
                                       double& D1) {
    double d[6];
#pragma unroll
    for (int m = 1; m < 6; ++m) d[m] = v[m] - v[m - 1];
    auto form = [&](double a, double b, double c, double B, double G, double D, double E, double Z) {
        const double y1 = fma(G, c, fma(B, b, a)), y2 = fma(E, c, b);
        double t = fma(Z * c, c, 1e-6 * 180.0 / 244.0);
        t = fma(y1, y1, fma(D * y2, y2, t));
        return t * t;
    };
    constexpr double kB = -1171.0 / 488, kG = 683.0 / 488, kD = 152295.0 / 238144, kE = -1.0 / 1, kZ = 45.0 / 61;
    constexpr double kB1 = -781.0 / 488, kG1 = 293.0 / 488, kD1 = 327975.0 / 238144, kE1 = -10153.0 / 21865, kZ1 = 91377.0 / 266753;
    qa = form(d[1], d[2], d[3], kB, kG, kD, kE, kZ);
    qb = form(d[2], d[3], d[4], kB1, kG1, kD1, kE1, kZ1);
    qc = form(d[5], d[4], d[3], kB, kG, kD, kE, kZ);
    D0 = fma(3.0, d[2] - d[3], d[4] - d[1]);
    D1 = fma(3.0, d[3] - d[4], d[5] - d[2]);
}

// a y- or z-pass: the ratios of the q_s by one division
__device__ __forceinline__ double weno_pass(const WenoX& w, const double (&v)[6]) {
    double qa, qb, qc, D0, D1;
    weno_q(v, qa, qb, qc, D0, D1);
    const double inv = inverse(qa * qc);
    const double ra = qb * qc * inv, rc = qb * qa * inv;
    const double pb = fma(w.L[3], v[4], fma(w.L[2], v[3], fma(w.L[1], v[2], w.L[0] * v[1])));
    const double den = fma(w.Cc, rc, fma(w.Ca, ra, w.Cb));
    return pb + div_newton(fma(w.Kc * rc, D1, w.Ka * ra * D0), den);
}

template <typename T, int TRACE, int WZ, int NZ>
__global__ void __launch_bounds__(WenoTile<T, WZ, NZ>::kThreads, 1)
    advect_phi_weno_tiled_kernel(GridView<T> src, T* __restrict__ out, Mac<T> mac, DtArg dt, T dx, T inv_dx,
                                 const __grid_constant__ BoxMap pmap) {
    using W = WenoTile<T, WZ, NZ>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* pbox = reinterpret_cast<T*>(align128(smem_raw));  // [z][y][x]
    const T* pb = pbox + 1;                              // the box from node tile - 3 along x
    // FP32: float4 entries {qa, qb, qc, 0} [row][floor index]; FP64: double2 entries, then D0 [row][kDiffs]
    void* const entries = pbox + W::kBoxN;
    __shared__ uint64_t bar;
    const int x0 = blockIdx.x * kWX, y0 = blockIdx.y * kWY, z0 = blockIdx.z * WZ;
    const int bx0 = x0 - 4, by0 = y0 - 3, bz0 = z0 - 3;
    const int tid = threadIdx.x + kWX * (threadIdx.y + kWY * threadIdx.z);
    const int lane = tid & 31, warp = tid >> 5;
    if (pmap.on) {
        if (tid == 0) {
            copy_boxes_begin(&bar, (unsigned)(W::kBoxN * sizeof(T)));
            tma_load_3d(pbox, &pmap.m, &bar, bx0, by0, bz0);
        }
    }
    // the thread's foot points while the box is on its way: their global reads are in flight together
    const int i = x0 + threadIdx.x, j = y0 + threadIdx.y;
    const bool column = i < src.n0 && j < src.n1;
    const T dtv = (T)dt_value(dt);
    // (FP32 keeps them in shared memory until their turn, for the registers of more warps)
    [[maybe_unused]] Vec3T<T> foot[sizeof(T) == 4 ? 1 : WZ / W::kNZ];
    [[maybe_unused]] float* const sfoot = reinterpret_cast<float*>(pbox + W::kBoxN) + W::kRows * W::kEP * 4 + tid;
#pragma unroll
    for (int q = 0; q < WZ / W::kNZ; ++q) {
        const int k = z0 + (int)threadIdx.z + q * W::kNZ;
        Vec3T<T> d{T(0), T(0), T(0)};
        if (column && k < src.n2)
            d = level_set_foot<T, TRACE>(cell_velocity(mac, i, j, k), i, j, k, dtv, dx, inv_dx,
                                         [&](const Axes<T>& a, const auto& far, auto) { return velocity_global(mac, a, far); });
        if constexpr (sizeof(T) == 4) {
            sfoot[q * W::kThreads] = d.x;
            sfoot[q * W::kThreads + W::kFoot] = d.y;
            sfoot[q * W::kThreads + 2 * W::kFoot] = d.z;
        } else {
            foot[q] = d;
        }
    }
    if (pmap.on) {
        __syncthreads();  // the mbarrier's initialisation is seen by every thread
        if (copy_boxes_failed(&bar, pmap.on == BOX_REPORTED)) {
            nan_column(src, out, x0 + threadIdx.x, y0 + threadIdx.y, z0, WZ);
            return;
        }
        AbsMax<T> unused;
        finish_box<T, kWNodes, kWBY, W::kBZ, false, W::kBX>(pbox, src, bx0, by0, bz0, unused);
    } else {
        for (int row = warp; row < W::kRows; row += W::kThreads / 32) {
            const int bz = row / kWBY, by = row - bz * kWBY;
            const int gy = clampi(by0 + by, 0, src.n1 - 1), gz = clampi(bz0 + bz, 0, src.n2 - 1);
            const T* p = src.d + (long long)src.n0 * (gy + (long long)src.n1 * gz);
            T* d = pbox + row * W::kBX;
            d[lane] = __ldg(p + clampi(bx0 + lane, 0, src.n0 - 1));
            if (lane < kWNodes - 32) d[32 + lane] = __ldg(p + clampi(bx0 + 32 + lane, 0, src.n0 - 1));
        }
    }
    __syncthreads();
    if constexpr (sizeof(T) == 4) {
        // two (row, floor index) entries a thread per pass in packed float2 arithmetic
        float4* q = static_cast<float4*>(entries);
        for (int e0 = tid; e0 < W::kEntries; e0 += 2 * W::kThreads) {
            const int e1 = e0 + W::kThreads < W::kEntries ? e0 + W::kThreads : e0;  // the tail repeats its entry
            const int r0 = e0 / kWBases, r1 = e1 / kWBases;
            const int b0 = e0 - r0 * kWBases, b1 = e1 - r1 * kWBases;
            const float* va = pb + r0 * W::kBX + b0;
            const float* vb = pb + r1 * W::kBX + b1;
            float2 v[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) v[m] = make_float2(va[m], vb[m]);
            float2 qa, qb, qc;
            weno6_sq2(v, qa, qb, qc);
            q[r0 * W::kEP + b0] = make_float4(qa.x, qb.x, qc.x, 0.f);
            if (e1 != e0) q[r1 * W::kEP + b1] = make_float4(qa.y, qb.y, qc.y, 0.f);
        }
    } else {
        double2* q = static_cast<double2*>(entries);
        double* D = reinterpret_cast<double*>(q + W::kRows * W::kEP);
        for (int e = tid; e < W::kEntries; e += W::kThreads) {
            const int row = e / kWBases, b = e - row * kWBases;
            const T* p = pb + row * W::kBX + b;
            const double v[6] = {p[0], p[1], p[2], p[3], p[4], p[5]};
            double qa, qb, qc, D0, D1;
            weno_q(v, qa, qb, qc, D0, D1);
            const double inv = inverse(qa * qc);
            q[e] = make_double2(qb * qc * inv, qb * qa * inv);
            D[row * W::kDiffs + b] = D0;
            if (b == kWBases - 1) D[row * W::kDiffs + b + 1] = D1;
        }
    }
    __syncthreads();
    if (!column) return;
#pragma unroll 1
    for (int n = 0; n < WZ / W::kNZ; ++n) {
        const int kk = (int)threadIdx.z + n * W::kNZ, k = z0 + kk;
        if (k >= src.n2) break;
        Vec3T<T> d;
        if constexpr (sizeof(T) == 4) {
            d = Vec3T<T>{sfoot[n * W::kThreads], sfoot[n * W::kThreads + W::kFoot], sfoot[n * W::kThreads + 2 * W::kFoot]};
        } else {
            d = foot[0];  // registers, not a dynamically indexed array
#pragma unroll
            for (int q = 1; q < WZ / W::kNZ; ++q) {
                d.x = n == q ? foot[q].x : d.x;
                d.y = n == q ? foot[q].y : d.y;
                d.z = n == q ? foot[q].z : d.z;
            }
        }
        d = foot_coords(d, dx, inv_dx);
        // stencil origin (floor - 2) relative to the box, per axis
        int px, py, pz;
        T fx, fy, fz;
        floor_index(d.x, px, fx);
        floor_index(d.y, py, fy);
        floor_index(d.z, pz, fz);
        px = (int)((unsigned)px + (unsigned)(foot_base<T>(i) - x0 + 1));
        py = (int)((unsigned)py + (unsigned)(foot_base<T>(j) - y0 + 1));
        pz = (int)((unsigned)pz + (unsigned)(foot_base<T>(k) - z0 + 1));
        T r = T(0);
        bool ok = false;
        // (within a cell of the four planes the sample lies in, whatever the tile: beyond, the global path)
        if ((unsigned)px < (unsigned)kWBases && (unsigned)py < (unsigned)(kWY + 2) && (unsigned)(pz - (kk & ~3)) < 6u) {
            if constexpr (sizeof(T) == 4) {
                // the x-passes of rows dj and dj + 1, and the y-passes of planes dk and dk + 1, together
                const float4* q = static_cast<const float4*>(entries);
                const WenoAxis<float> wx = weno_axis(fx), wy = weno_axis(fy);
                float zl[6];
#pragma unroll
                for (int dk = 0; dk < 6; dk += 2) {
                    float2 yl[6];  // .x: plane dk, .y: plane dk + 1
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int row0 = (pz + dk + u) * kWBY + py;
#pragma unroll
                        for (int dj = 0; dj < 6; dj += 2) {
                            const float* va = pb + (row0 + dj) * W::kBX + px;
                            const float* vb = va + W::kBX;
                            const float4 ea = q[(row0 + dj) * W::kEP + px], eb = q[(row0 + dj + 1) * W::kEP + px];
                            float2 v[6];
#pragma unroll
                            for (int m = 0; m < 6; ++m) v[m] = make_float2(va[m], vb[m]);
                            const float2 y = weno6_combine2(wx, v, make_float2(ea.x, eb.x), make_float2(ea.y, eb.y),
                                                            make_float2(ea.z, eb.z));
                            if (u == 0) {
                                yl[dj].x = y.x;
                                yl[dj + 1].x = y.y;
                            } else {
                                yl[dj].y = y.x;
                                yl[dj + 1].y = y.y;
                            }
                        }
                    }
                    const float2 zv = weno6_eval2(wy, yl);
                    zl[dk] = zv.x;
                    zl[dk + 1] = zv.y;
                }
                r = weno6_eval(weno_axis(fz), zl[0], zl[1], zl[2], zl[3], zl[4], zl[5]);
                ok = true;
            } else {
                const WenoX wx = weno_x(fx), wy = weno_x(fy);
                const double2* q = static_cast<const double2*>(entries);
                const double* D = reinterpret_cast<const double*>(q + W::kRows * W::kEP);
                double zl[6];
#pragma unroll
                for (int dk = 0; dk < 6; ++dk) {
                    const int row0 = (pz + dk) * kWBY + py;
                    double yl[6];
#pragma unroll
                    for (int dj = 0; dj < 6; ++dj) {
                        const int row = row0 + dj;
                        const T* v = pb + row * W::kBX + px;
                        const double2 e = q[row * kWBases + px];
                        const double* dd = D + row * W::kDiffs + px;
                        const double p = fma(wx.L[3], v[4], fma(wx.L[2], v[3], fma(wx.L[1], v[2], wx.L[0] * v[1])));
                        const double den = fma(wx.Cc, e.y, fma(wx.Ca, e.x, wx.Cb));
                        yl[dj] = p + div_newton(fma(wx.Kc * e.y, dd[1], wx.Ka * e.x * dd[0]), den);
                    }
                    const double zv = weno_pass(wy, yl);
                    // registers, not a dynamically indexed array
                    zl[0] = dk == 0 ? zv : zl[0];
                    zl[1] = dk == 1 ? zv : zl[1];
                    zl[2] = dk == 2 ? zv : zl[2];
                    zl[3] = dk == 3 ? zv : zl[3];
                    zl[4] = dk == 4 ? zv : zl[4];
                    zl[5] = dk == 5 ? zv : zl[5];
                }
                r = weno_pass(weno_x(fz), zl);
                ok = isfinite(r);
            }
        }
        if (!ok) r = sample_weno6(src, foot_base<T>(i), foot_base<T>(j), foot_base<T>(k), d.x, d.y, d.z);
        const int oc = cell_index(src, i, j, k);
        if (EL_IN(oc, (long long)src.n0 * src.n1 * src.n2, 3)) out[oc] = r;
    }
}

// Grid views of the scene's grids (staggered_grid.h:100-112): comp 0 = cells, 1/2/3 = u/v/w.
template <typename T>
GridView<T> make_view(const void* d, int ni, int nj, int nk, int comp) {
    return GridView<T>{static_cast<const T*>(d), ni + (comp == 1), nj + (comp == 2), nk + (comp == 3)};
}

template <typename T, int TRACE, int SAMPLE>
static void launch_one(const GridView<T>& src, int comp, void* out, const Mac<T>& mac, DtArg dt, T dx, int rows,
                       cudaStream_t s) {
    dim3 block(32, rows, 1);
    dim3 grid((src.n0 + 31) / 32, (src.n1 + rows - 1) / rows, src.n2);
    advect_kernel<T, TRACE, SAMPLE><<<grid, block, 0, s>>>(src, comp, static_cast<T*>(out), mac, dt, dx,
                                                           T(1) / dx);
}

template <typename T>
static void launch_dispatch(const GridView<T>& src, int comp, void* out, const Mac<T>& mac, DtArg dt, T dx,
                            int trace, int sample, int rows, cudaStream_t s) {
    if (trace == EL_TRACE_RK2 && sample == EL_SAMPLE_TRILINEAR)
        launch_one<T, EL_TRACE_RK2, EL_SAMPLE_TRILINEAR>(src, comp, out, mac, dt, dx, rows, s);
    else if (trace == EL_TRACE_RK2 && sample == EL_SAMPLE_WENO6)
        launch_one<T, EL_TRACE_RK2, EL_SAMPLE_WENO6>(src, comp, out, mac, dt, dx, rows, s);
    else if (trace == EL_TRACE_RK3 && sample == EL_SAMPLE_TRILINEAR)
        launch_one<T, EL_TRACE_RK3, EL_SAMPLE_TRILINEAR>(src, comp, out, mac, dt, dx, rows, s);
    else
        launch_one<T, EL_TRACE_RK3, EL_SAMPLE_WENO6>(src, comp, out, mac, dt, dx, rows, s);
}

// Launch the advection of `which` (0 = cell-centred grid `in`, 1..3 = face component) into out.
// Returns the number of kernels launched.
template <typename T>
static int advect_launch(int ni, int nj, int nk, double dx_d, int comp, void* out, const void* in,
                         const void* vu, const void* vv, const void* vw, DtArg dt, int trace,
                         int sample, int rows, cudaStream_t s) {
    const T dx = (T)dx_d;
    Mac<T> mac{make_view<T>(vu, ni, nj, nk, 1), make_view<T>(vv, ni, nj, nk, 2),
               make_view<T>(vw, ni, nj, nk, 3)};
    GridView<T> src = make_view<T>(in, ni, nj, nk, comp);
    launch_dispatch<T>(src, comp, out, mac, dt, dx, trace, sample, rows, s);
    return 1;
}

// The box map of one array for boxes of bx x by x bz (BOX_NONE when copies are off or the
// array's pitch or address does not allow them: the kernel then stages it by plain loads).
template <typename T>
static BoxMap box_map(const GridView<T>& g, BoxCopies copy, unsigned bx, unsigned by, unsigned bz) {
    BoxMap b;
    std::memset(&b, 0, sizeof(b));
    if (copy != BOX_NONE &&
        tma_encode_3d(&b.m, sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                      (int)sizeof(T), g.d, g.n0, g.n1, g.n2, g.n0, bx, by, bz))
        b.on = copy;
    return b;
}

template <typename T>
static MacMaps mac_maps(const Mac<T>& mac, BoxCopies copy) {
    MacMaps m;
    m.c[0] = box_map(mac.u, copy, kBoxX, kBoxY, kBoxZ);
    m.c[1] = box_map(mac.v, copy, kBoxX, kBoxY, kBoxZ);
    m.c[2] = box_map(mac.w, copy, kBoxX, kBoxY, kBoxZ);
    return m;
}

// the tiled kernels: the level set (any scheme), and the velocity advecting itself (trilinear);
// dynamic shared memory holds the boxes plus 128 bytes to align them
template <typename T, int TRACE>
static int launch_phi_tiled(const GridView<T>& src, void* out, const Mac<T>& mac, DtArg dt, T dx, BoxCopies copy,
                            cudaStream_t s) {
    const int smem = 3 * kBoxN * (int)sizeof(T) + 128;
    if (cudaFuncSetAttribute(advect_phi_tiled_kernel<T, TRACE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) != cudaSuccess) {
        cudaGetLastError();  // the per-sample kernel takes over: not an error of the call
        return -1;
    }
    const dim3 grid((src.n0 + kTileX - 1) / kTileX, (src.n1 + kTileY - 1) / kTileY, (src.n2 + kTileZ - 1) / kTileZ);
    advect_phi_tiled_kernel<T, TRACE><<<grid, dim3(kTileX, kTileY, 1), smem, s>>>(
        src, static_cast<T*>(out), mac, dt, dx, T(1) / dx, mac_maps(mac, copy));
    return 1;
}

template <typename T, int TRACE, int WZ, int NZ>
static int launch_phi_weno_tile(const GridView<T>& src, void* out, const Mac<T>& mac, DtArg dt, T dx, BoxCopies copy,
                                cudaStream_t s) {
    using W = WenoTile<T, WZ, NZ>;
    const int smem = W::kBytes + 128;
    if (cudaFuncSetAttribute(advect_phi_weno_tiled_kernel<T, TRACE, WZ, NZ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) != cudaSuccess) {
        cudaGetLastError();  // the per-sample kernel takes over: not an error of the call
        return -1;
    }
    const dim3 grid((src.n0 + kWX - 1) / kWX, (src.n1 + kWY - 1) / kWY, (src.n2 + WZ - 1) / WZ);
    advect_phi_weno_tiled_kernel<T, TRACE, WZ, NZ><<<grid, dim3(kWX, kWY, W::kNZ), smem, s>>>(
        src, static_cast<T*>(out), mac, dt, dx, T(1) / dx, box_map(src, copy, W::kBX, kWBY, W::kBZ));
    return 1;
}

// FP32: a CTA of 1024 threads per tile, four planes at a time.  Tiles of eight planes form 3.7
// entries a sample against 5.5 of four planes (256^3: 1436 against 1569 us; 151 x 97 x 133: 216
// against 232); where every tile of four planes has an SM of its own, those finish sooner (48^3:
// 25.2 against 39.6 us), and so where the grid has no more planes (300 x 300 x 1: 37.9 against 42; 300 x
// 300 x 2: 48.5).  512 threads a tile took 1453 us at 256^3, 768 on six planes 1449.
static int device_sms() {
    int dev = 0, sms = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
                   cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess
               ? sms
               : 1;
}

template <typename T, int TRACE>
static int launch_phi_weno_tiled(const GridView<T>& src, void* out, const Mac<T>& mac, DtArg dt, T dx, BoxCopies copy,
                                 cudaStream_t s) {
    if constexpr (sizeof(T) == 4) {
        const long long tiles4 = (long long)((src.n0 + kWX - 1) / kWX) * ((src.n1 + kWY - 1) / kWY) * ((src.n2 + 3) / 4);
        if (src.n2 > 4 && tiles4 > device_sms()) return launch_phi_weno_tile<T, TRACE, 8, 4>(src, out, mac, dt, dx, copy, s);
        return launch_phi_weno_tile<T, TRACE, 4, 4>(src, out, mac, dt, dx, copy, s);
    } else {
        return launch_phi_weno_tile<T, TRACE, 4, 1>(src, out, mac, dt, dx, copy, s);
    }
}

template <typename T, int TRACE>
static int launch_velocity_tiled(const Mac<T>& mac, void* ou, void* ov, void* ow, DtArg dt, T dx, BoxCopies copy,
                                 cudaStream_t s) {
    const int smem = 3 * kBoxN * (int)sizeof(T) + 128;
    if (cudaFuncSetAttribute(advect_velocity_tiled_kernel<T, TRACE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) != cudaSuccess) {
        cudaGetLastError();  // the per-sample kernel takes over: not an error of the call
        return -1;
    }
    // tiles of cells
    const dim3 grid((mac.v.n0 + kTileX - 1) / kTileX, (mac.u.n1 + kTileY - 1) / kTileY,
                    (mac.u.n2 + kTileZ - 1) / kTileZ);
    advect_velocity_tiled_kernel<T, TRACE><<<grid, dim3(kTileX, kTileY, 1), smem, s>>>(
        mac, static_cast<T*>(ou), static_cast<T*>(ov), static_cast<T*>(ow), dt, T(1) / dx, mac_maps(mac, copy));
    return 1;
}

template <typename T>
static int advect_phi_tiled_t(int ni, int nj, int nk, double dx_d, void* out, const void* in, const void* vu,
                              const void* vv, const void* vw, DtArg dt, int trace, int sample, BoxCopies copy,
                              cudaStream_t s) {
    const T dx = (T)dx_d;
    Mac<T> mac{make_view<T>(vu, ni, nj, nk, 1), make_view<T>(vv, ni, nj, nk, 2),
               make_view<T>(vw, ni, nj, nk, 3)};
    GridView<T> src = make_view<T>(in, ni, nj, nk, 0);
    if (sample == EL_SAMPLE_WENO6)
        return trace == EL_TRACE_RK2 ? launch_phi_weno_tiled<T, EL_TRACE_RK2>(src, out, mac, dt, dx, copy, s)
                                     : launch_phi_weno_tiled<T, EL_TRACE_RK3>(src, out, mac, dt, dx, copy, s);
    if (trace == EL_TRACE_RK2)
        return launch_phi_tiled<T, EL_TRACE_RK2>(src, out, mac, dt, dx, copy, s);
    return launch_phi_tiled<T, EL_TRACE_RK3>(src, out, mac, dt, dx, copy, s);
}

template <typename T>
static int advect_velocity_tiled_t(int ni, int nj, int nk, double dx_d, void* ou, void* ov, void* ow, const void* vu,
                                   const void* vv, const void* vw, DtArg dt, int trace, BoxCopies copy, cudaStream_t s) {
    const T dx = (T)dx_d;
    Mac<T> mac{make_view<T>(vu, ni, nj, nk, 1), make_view<T>(vv, ni, nj, nk, 2),
               make_view<T>(vw, ni, nj, nk, 3)};
    if (trace == EL_TRACE_RK2) return launch_velocity_tiled<T, EL_TRACE_RK2>(mac, ou, ov, ow, dt, dx, copy, s);
    return launch_velocity_tiled<T, EL_TRACE_RK3>(mac, ou, ov, ow, dt, dx, copy, s);
}

// Level set through the tiled kernel; returns kernels launched, -1 on a launch set-up failure.
// copy: stage the boxes by box copies where the arrays allow it (else plain loads throughout).
int advect_phi_tiled(int dtype, int ni, int nj, int nk, double dx, void* out, const void* in, const void* vu,
                     const void* vv, const void* vw, const Scalars* dts, double dtv, int trace, int sample, BoxCopies copy,
                     cudaStream_t s) {
    DtArg dt{dts, dtv};
    if (dtype == EL_F64)
        return advect_phi_tiled_t<double>(ni, nj, nk, dx, out, in, vu, vv, vw, dt, trace, sample, copy, s);
    return advect_phi_tiled_t<float>(ni, nj, nk, dx, out, in, vu, vv, vw, dt, trace, sample, copy, s);
}

// u, v, w advected through themselves with trilinear sampling, one tiled launch
int advect_velocity_tiled(int dtype, int ni, int nj, int nk, double dx, void* ou, void* ov, void* ow, const void* vu,
                          const void* vv, const void* vw, const Scalars* dts, double dtv, int trace, BoxCopies copy,
                          cudaStream_t s) {
    DtArg dt{dts, dtv};
    if (dtype == EL_F64)
        return advect_velocity_tiled_t<double>(ni, nj, nk, dx, ou, ov, ow, vu, vv, vw, dt, trace, copy, s);
    return advect_velocity_tiled_t<float>(ni, nj, nk, dx, ou, ov, ow, vu, vv, vw, dt, trace, copy, s);
}

// the box-copy wait fault word, read and cleared (synchronises the device)
bool advect_fault_take() {
    unsigned v = 0, z = 0;
    if (cudaMemcpyFromSymbol(&v, advect_wait_fault, sizeof(v)) != cudaSuccess) return false;
    if (v) cudaMemcpyToSymbol(advect_wait_fault, &z, sizeof(z));
    return v != 0;
}

int advect_any(int dtype, int ni, int nj, int nk, double dx, int comp, void* out, const void* in,
               const void* vu, const void* vv, const void* vw, const Scalars* dts, double dtv,
               int trace, int sample, cudaStream_t s, int rows) {
    DtArg dt{dts, dtv};
    rows = (rows == 1 || rows == 2 || rows == 8) ? rows : 4;
    if (dtype == EL_F64)
        return advect_launch<double>(ni, nj, nk, dx, comp, out, in, vu, vv, vw, dt, trace, sample, rows, s);
    return advect_launch<float>(ni, nj, nk, dx, comp, out, in, vu, vv, vw, dt, trace, sample, rows, s);
}

EL_CHECK_EXPORT(advect)

}  // namespace el
