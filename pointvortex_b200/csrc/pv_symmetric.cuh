// pv_symmetric.cuh — warp tiles evaluated once per unordered pair (box, plane, disk),
// shared by the single-simulation kernels (pv_symmetric.cu) and the batched ensembles
// (pv_batch.cu).
//
// A tile is 32 targets (one per lane) against 32 sources. The reactions that the sources
// accumulate rotate one lane per step by shuffles; after 32 steps every (target, source) pair has
// been met once and every reaction is back in its home lane. What a pair's two terms have in
// common is evaluated once: in the box and the plane everything but the circulation and the sign,
// in the disk the two reciprocals. Callers pass the scaled circulations times the policy's kScale
// (PeriodicSym's terms carry half sines: 2 * Gamma * 0.5/L).
#pragma once

#include "pv_geometry.cuh"
#include "pv_pair32.cuh"

namespace pvb {
namespace sym {

__device__ __forceinline__ double rotate(double v, int from) {
    return __shfl_sync(0xffffffffu, v, from);
}

// One vortex of a tile: position and the scaled circulation times the policy's kScale.
struct Vortex {
    double x, y, g;
};

// What the geometries evaluated this way provide:
//   react<NEAR>(g, t, s, u, v, ru, rv): a pair's terms, the target's into (u, v) and the source's
//     into (ru, rv). NEAR: all vortices of the tile satisfy near() (kNearForm policies only);
//   one(g, t, s, u, v): the target's alone; self(g, t, u, v): what a vortex does to itself.
//
// The box and the plane have antisymmetric kernels K: the target's velocity changes by u -= c_s K_u,
// v += c_s K_v and the source's by u += c_t K_u, v -= c_t K_v.
template <class K> struct Antisymmetric {
    static constexpr bool kNearForm = false;
    static constexpr double kScale = 1.0;
    __device__ __forceinline__ static bool near(const GeometryConsts &, double, double) {
        return false;
    }
    template <bool NEAR>
    __device__ __forceinline__ static void react(const GeometryConsts &g, const Vortex &t,
                                                 const Vortex &s, double &u, double &v, double &ru,
                                                 double &rv) {
        double ku, kv;
        if constexpr (NEAR)
            K::values_near(g, t.x, t.y, s.x, s.y, ku, kv);
        else
            K::values(g, t.x, t.y, s.x, s.y, ku, kv);
        u = fma(-s.g, ku, u);
        v = fma(s.g, kv, v);
        ru = fma(t.g, ku, ru);
        rv = fma(-t.g, kv, rv);
    }
    __device__ __forceinline__ static void one(const GeometryConsts &g, const Vortex &t,
                                               const Vortex &s, double &u, double &v) {
        double ku, kv;
        K::values(g, t.x, t.y, s.x, s.y, ku, kv);
        u = fma(-s.g, ku, u);
        v = fma(s.g, kv, v);
    }
    // the reference skips the self pair (and in the periodic box it contributes exactly 0)
    __device__ __forceinline__ static void self(const GeometryConsts &, const Vortex &, double &,
                                                double &) {}
};

struct PeriodicSym : Antisymmetric<PeriodicSym> {
    // the terms carry half sines (PeriodicPair::terms<true>): circulations are doubled
    static constexpr double kScale = 2.0;
    __device__ __forceinline__ static void values(const GeometryConsts &g, double tx, double ty,
                                                  double sx, double sy, double &ku, double &kv) {
        double au, bu, av, bv;
        PeriodicPair::terms<true>(g, tx, ty, sx, sy, au, bu, av, bv);
        ku = au * rcp_refined(bu);
        kv = av * rcp_refined(bv);
    }
};

// The box from six images up (ZetaPair). Tiles whose vortices are all in or near the box reduce a
// difference by one subtraction (values_near): two FP64 instructions an axis with it, four without
// (a population that has drifted out of the box: 8 % more of the pair's 50).
template <class Z> struct ZetaSymT : Antisymmetric<ZetaSymT<Z>> {
    static constexpr bool kNearForm = true;
    __device__ __forceinline__ static void values(const GeometryConsts &g, double tx, double ty,
                                                  double sx, double sy, double &ku, double &kv) {
        Z::terms(g, Z::reduce(g, tx - sx, g.lx, g.inv_lx), Z::reduce(g, ty - sy, g.ly, g.inv_ly), ku,
                 kv);
    }
    __device__ __forceinline__ static void values_near(const GeometryConsts &g, double tx,
                                                       double ty, double sx, double sy,
                                                       double &ku, double &kv) {
        Z::terms(g, Z::reduce_near(g, tx - sx, g.lx), Z::reduce_near(g, ty - sy, g.ly), ku, kv);
    }
    __device__ __forceinline__ static bool near(const GeometryConsts &g, double x, double y) {
        return Z::inside(g, x, y);
    }
};
using ZetaSym = ZetaSymT<ZetaPair>;
using ZetaUnitSym = ZetaSymT<ZetaUnitPair>;

// The infinite plane (InfinitePair): K = (dy, dx) / (r^2 + eps^2), exactly odd in (dx, dy).
struct PlaneSym : Antisymmetric<PlaneSym> {
    __device__ __forceinline__ static void values(const GeometryConsts &g, double tx, double ty,
                                                  double sx, double sy, double &ku, double &kv) {
        const double dx = tx - sx, dy = ty - sy;
        const double inv = rcp_refined(fma(dx, dx, fma(dy, dy, g.eps2)));
        ku = dy * inv;
        kv = dx * inv;
    }
};

// The disk (DiskPair). The direct term is the plane's. For the wall images, with A = R^2 - t.s and
// B = t x s (t_y s_x - t_x s_y), the target gets c_s (B s_x - A s_y, A s_x + B s_y) / (A^2 + B^2):
// exchanging the vortices keeps A and negates B, so one reciprocal serves both sides. Beside the
// circulations stand the moments c s and c t. 34 FP64 instructions an unordered pair (two of them
// the source's moments, shared by the lane's targets) against 58 for its two ordered pairs;
// measured per launch, ordered against this: N = 4096 43 -> 36 us, 8192 135 -> 100 us, 12 000
// 294 -> 185 us, 16 384 504 -> 314 us, 40 000 2756 -> 1772 us. The FP64 pipe bounds it: 34
// instructions of two or (18, all operands distinct registers) three cycles.
struct DiskSym {
    static constexpr bool kNearForm = false;
    static constexpr double kScale = 1.0;
    __device__ __forceinline__ static bool near(const GeometryConsts &, double, double) {
        return false;
    }
    // (A, B) / (A^2 + B^2)
    __device__ __forceinline__ static void image(const GeometryConsts &g, const Vortex &t,
                                                 const Vortex &s, double &a, double &b) {
        const double A = fma(-t.y, s.y, fma(-t.x, s.x, g.radius2));
        const double B = fma(t.y, s.x, -t.x * s.y);
        const double inv = rcp_refined(fma(A, A, B * B));
        a = A * inv;
        b = B * inv;
    }
    template <bool NEAR>
    __device__ __forceinline__ static void react(const GeometryConsts &g, const Vortex &t,
                                                 const Vortex &s, double &u, double &v, double &ru,
                                                 double &rv) {
        const double dx = t.x - s.x, dy = t.y - s.y;
        const double inv = rcp_refined(fma(dx, dx, dy * dy));
        const double ku = dy * inv, kv = dx * inv;
        double a, b;
        image(g, t, s, a, b);
        const double smx = s.g * s.x, smy = s.g * s.y, tmx = t.g * t.x, tmy = t.g * t.y;
        u = fma(-s.g, ku, u);
        ru = fma(t.g, ku, ru);
        v = fma(s.g, kv, v);
        rv = fma(-t.g, kv, rv);
        u = fma(b, smx, u);
        v = fma(b, smy, v);
        ru = fma(-b, tmx, ru);
        rv = fma(-b, tmy, rv);
        u = fma(-a, smy, u);
        v = fma(a, smx, v);
        ru = fma(-a, tmy, ru);
        rv = fma(a, tmx, rv);
    }
    __device__ __forceinline__ static void one(const GeometryConsts &g, const Vortex &t,
                                               const Vortex &s, double &u, double &v) {
        const double dx = t.x - s.x, dy = t.y - s.y;
        const double c = s.g * rcp_refined(fma(dx, dx, dy * dy));
        u = fma(-c, dy, u);
        v = fma(c, dx, v);
        self_image(g, t, s, u, v);
    }
    __device__ __forceinline__ static void self_image(const GeometryConsts &g, const Vortex &t,
                                                      const Vortex &s, double &u, double &v) {
        double a, b;
        image(g, t, s, a, b);
        const double smx = s.g * s.x, smy = s.g * s.y;
        u = fma(b, smx, fma(-a, smy, u));
        v = fma(a, smx, fma(b, smy, v));
    }
    // a vortex meets its own image
    __device__ __forceinline__ static void self(const GeometryConsts &g, const Vortex &t, double &u,
                                                double &v) {
        self_image(g, t, t, u, v);
    }
};

// Target t against the sources held in the lanes (s and their reactions ru, rv); adds the targets'
// sums to u, v and the sources' to ru, rv. Sources end at home. FULL: all 32 targets and sources
// exist, no predicates.
template <class P, bool FULL>
__device__ __forceinline__ void react_tile_t(const GeometryConsts &g, const Vortex &t, bool t_ok,
                                             Vortex s, int s_ok, double &u, double &v, double &ru,
                                             double &rv) {
    const int next = (threadIdx.x + 1) & 31;
#pragma unroll 2
    for (int k = 0; k < 32; ++k) {
        if (FULL || (t_ok && s_ok))
            P::template react<false>(g, t, s, u, v, ru, rv);
        s.x = rotate(s.x, next);
        s.y = rotate(s.y, next);
        s.g = rotate(s.g, next);
        ru = rotate(ru, next);
        rv = rotate(rv, next);
        if (!FULL)
            s_ok = __shfl_sync(0xffffffffu, s_ok, next);
    }
}

// The sources of a tile in the warp's shared buffer, each twice, 32 entries apart, so that step k of
// lane l reads entry l + k without a wrap.
struct SourceBuffer {
    double2 xy[64];
    double g[64];
    __device__ __forceinline__ void fill(const Vortex &s) {
        const int lane = threadIdx.x & 31;
        __syncwarp();  // the previous tile's reads are done
        xy[lane] = xy[lane + 32] = make_double2(s.x, s.y);
        g[lane] = g[lane + 32] = s.g;
        __syncwarp();
    }
};

// T targets per lane (T sub-blocks of targets) against the 32 sources of the buffer, every target
// and source present. Only the reactions rotate (two double shuffles a step, shared by the T
// pairs); reading the sources instead of rotating them too (five) is 6 % faster with the box's
// terms (N = 16384, T = 1: 500 against 532 us; T = 2: 472 against 493 us). U steps are unrolled:
// two with one target per lane, four with two, none with four (the disk at N = 16384: 314 against
// 325 us unrolled by two).
template <class P, int T, bool NEAR, int U = (T == 2 ? 4 : T == 4 ? 1 : 2)>
__device__ __forceinline__ void react_tiles_steps(const GeometryConsts &g, const Vortex (&t)[T],
                                                  const SourceBuffer &b, double (&u)[T],
                                                  double (&v)[T], double &ru, double &rv) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
    const double2 *xy = b.xy + lane;
    const double *sgs = b.g + lane;
#pragma unroll U
    for (int k = 0; k < 32; ++k) {
        const Vortex s = {xy[k].x, xy[k].y, sgs[k]};
#pragma unroll
        for (int q = 0; q < T; ++q)
            P::template react<NEAR>(g, t[q], s, u[q], v[q], ru, rv);
        ru = rotate(ru, next);
        rv = rotate(rv, next);
    }
}

// The same with the sources rotating through the lanes beside their reactions. With eight targets
// per lane (the plane's wide form) the shuffles of a step are shared by eight pairs, and reading
// the sources instead is slower: launches of 1204 against 1175 us at N = 50 001, 1919 against
// 1892 us at 65 536.
template <class P, int T>
__device__ __forceinline__ void react_tiles_rotating(const GeometryConsts &g,
                                                     const Vortex (&t)[T], Vortex s,
                                                     double (&u)[T], double (&v)[T], double &ru,
                                                     double &rv) {
    const int next = (threadIdx.x + 1) & 31;
#pragma unroll 2
    for (int k = 0; k < 32; ++k) {
#pragma unroll
        for (int q = 0; q < T; ++q)
            P::template react<false>(g, t[q], s, u[q], v[q], ru, rv);
        s.x = rotate(s.x, next);
        s.y = rotate(s.y, next);
        s.g = rotate(s.g, next);
        ru = rotate(ru, next);
        rv = rotate(rv, next);
    }
}

// One whole tile set of T targets per lane. near: this lane's targets satisfy P::near.
template <class P, int T, bool BUFFERED>
__device__ __forceinline__ void react_tiles_full(const GeometryConsts &g, const Vortex (&t)[T],
                                                 const Vortex &s, SourceBuffer &b, bool near,
                                                 double (&u)[T], double (&v)[T], double &ru,
                                                 double &rv) {
    if constexpr (!BUFFERED) {
        react_tiles_rotating<P, T>(g, t, s, u, v, ru, rv);
        return;
    }
    b.fill(s);
    if constexpr (P::kNearForm) {
        if (__all_sync(0xffffffffu, near && P::near(g, s.x, s.y))) {
            react_tiles_steps<P, T, true>(g, t, b, u, v, ru, rv);
            return;
        }
    }
    react_tiles_steps<P, T, false>(g, t, b, u, v, ru, rv);
}

// Target side only. same_block: the sources are the targets' own lanes, so step 0 is the vortex
// itself.
template <class P>
__device__ __forceinline__ void one_sided_tile(const GeometryConsts &g, const Vortex &t, bool t_ok,
                                               Vortex s, int s_ok, bool same_block, double &u,
                                               double &v) {
    const int next = (threadIdx.x + 1) & 31;
    for (int k = 0; k < 32; ++k) {
        if (t_ok && s_ok && !(same_block && k == 0))
            P::one(g, t, s, u, v);
        s.x = rotate(s.x, next);
        s.y = rotate(s.y, next);
        s.g = rotate(s.g, next);
        s_ok = __shfl_sync(0xffffffffu, s_ok, next);
    }
    if (same_block && t_ok)
        P::self(g, t, u, v);
}

// FP32-compensated tiles: the 32 sources (hi/lo coordinates and FP32 circulation) sit in this
// warp's shared buffer, read at index (lane + k) & 31; only their FP32 reactions rotate through
// the lanes. V: the pair kernel (f32::Periodic32, f32::Plane32). The callers promote the FP32
// sums of each tile into FP64.
//
// Near pairs (V::kNear kernels) contribute 0 here and are listed for the FP64 pass, in both
// directions, under the lane's target `ti` and the tile's source j0 + j.
struct NearTile {
    f32::NearLists lists;  // lists.count == nullptr: no near field
    size_t ti;             // this lane's target
    size_t j0;             // the tile's first source
};

template <class V>
__device__ __forceinline__ void list_near_pair(const NearTile &nt, int j, bool both) {
    if (V::kNear && nt.lists.count) {
        f32::near_append(nt.lists, nt.ti, static_cast<unsigned>(nt.j0 + j));
        if (both)
            f32::near_append(nt.lists, nt.j0 + j, static_cast<unsigned>(nt.ti));
    }
}

template <class V, bool FULL>
__device__ __forceinline__ void react_tile32_t(const f32::F32Geometry &f, const float4 t, float tg,
                                               bool t_ok, const float4 *sf, const float *sg,
                                               int s_count, float &u, float &v, float &ru,
                                               float &rv, const NearTile &nt) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
#pragma unroll 2
    for (int k = 0; k < 32; ++k) {
        const int j = (lane + k) & 31;
        if (FULL || (t_ok && j < s_count)) {
            float ku, kv;
            if (V::values(f, t, sf[j], ku, kv))
                list_near_pair<V>(nt, j, true);
            const float g = sg[j];
            u = fmaf(-g, ku, u);
            v = fmaf(g, kv, v);
            ru = fmaf(tg, ku, ru);
            rv = fmaf(-tg, kv, rv);
        }
        ru = __shfl_sync(0xffffffffu, ru, next);
        rv = __shfl_sync(0xffffffffu, rv, next);
    }
}

template <class V = f32::Periodic32>
__device__ __forceinline__ void react_tile32(const f32::F32Geometry &f, const float4 t, float tg,
                                             bool t_ok, const float4 *sf, const float *sg,
                                             int s_count, float &u, float &v, float &ru,
                                             float &rv, const NearTile &nt) {
    if (__all_sync(0xffffffffu, t_ok && s_count == 32))
        react_tile32_t<V, true>(f, t, tg, t_ok, sf, sg, s_count, u, v, ru, rv, nt);
    else
        react_tile32_t<V, false>(f, t, tg, t_ok, sf, sg, s_count, u, v, ru, rv, nt);
}

// The sources of a whole tile packed for zeta_values32_x2: entry j holds source j & 31 and, in the
// other f32x2 lane, source (j + 16) & 31, so that step k of lane l (k < 16) reads entry l + k and
// meets both. Coordinates negated.
struct SourceBuffer32 {
    float4 hi[48];  // (-xh_j, -xh_j+16, -yh_j, -yh_j+16)
    float4 lo[48];
    float4 g[48];   // (-g_j, -g_j+16, g_j, g_j+16)
    __device__ __forceinline__ void fill(const float4 s, float sg) {
        const int lane = threadIdx.x & 31;
        float4 o;
        o.x = __shfl_xor_sync(0xffffffffu, s.x, 16);
        o.y = __shfl_xor_sync(0xffffffffu, s.y, 16);
        o.z = __shfl_xor_sync(0xffffffffu, s.z, 16);
        o.w = __shfl_xor_sync(0xffffffffu, s.w, 16);
        const float og = __shfl_xor_sync(0xffffffffu, sg, 16);
        const float4 h = make_float4(-s.x, -o.x, -s.y, -o.y), l = make_float4(-s.z, -o.z, -s.w, -o.w);
        __syncwarp();  // the previous tile's reads are done
        hi[lane] = h;
        lo[lane] = l;
        const float4 gg = make_float4(-sg, -og, sg, og);
        g[lane] = gg;
        if (lane < 16) {
            hi[lane + 32] = h;
            lo[lane + 32] = l;
            g[lane + 32] = gg;
        }
        __syncwarp();
    }
};

// A whole tile of 32 targets and the buffer's 32 sources in 16 steps of two pairs a lane. Each FP32
// sum covers 16 terms; a target's two (one a lane of the pair) and a source's two are added in FP64.
__device__ __forceinline__ void react_tile_zeta32(const f32::F32Geometry &f, const float4 t,
                                                  float tg, const SourceBuffer32 &b, double &ud,
                                                  double &vd, double &rud, double &rvd,
                                                  const NearTile &nt) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
    const float2 thx = f32::splat2(t.x), thy = f32::splat2(t.y), tlx = f32::splat2(t.z),
                 tly = f32::splat2(t.w), tg2 = f32::splat2(tg), tgm2 = f32::splat2(-tg);
    float2 u = f32::splat2(0.0f), v = u, ru = u, rv = u;
#pragma unroll 2
    for (int k = 0; k < 16; ++k) {
        const float4 h = b.hi[lane + k], l = b.lo[lane + k];
        const float4 g = b.g[lane + k];
        float2 ku, kv;
        bool near0, near1;
        f32::zeta_values32_x2(f, thx, thy, tlx, tly, make_float2(h.x, h.y), make_float2(h.z, h.w),
                              make_float2(l.x, l.y), make_float2(l.z, l.w), ku, kv, near0, near1);
        if (near0 || near1) {
            if (near0)
                list_near_pair<f32::Periodic32>(nt, (lane + k) & 31, true);
            if (near1)
                list_near_pair<f32::Periodic32>(nt, (lane + k + 16) & 31, true);
        }
        u = f32::fma2(make_float2(g.x, g.y), ku, u);
        v = f32::fma2(make_float2(g.z, g.w), kv, v);
        ru = f32::fma2(tg2, ku, ru);
        rv = f32::fma2(tgm2, kv, rv);
        ru.x = __shfl_sync(0xffffffffu, ru.x, next);
        ru.y = __shfl_sync(0xffffffffu, ru.y, next);
        rv.x = __shfl_sync(0xffffffffu, rv.x, next);
        rv.y = __shfl_sync(0xffffffffu, rv.y, next);
    }
    ud += static_cast<double>(u.x) + static_cast<double>(u.y);
    vd += static_cast<double>(v.x) + static_cast<double>(v.y);
    // after 16 rotations lane l holds source l's second sum and source l + 16's first
    rud += static_cast<double>(ru.y) +
           static_cast<double>(__shfl_xor_sync(0xffffffffu, ru.x, 16));
    rvd += static_cast<double>(rv.y) +
           static_cast<double>(__shfl_xor_sync(0xffffffffu, rv.x, 16));
}

// T targets per lane against the 32 sources of the buffer, every target and source present: each
// step serves T pairs per lane, and the reactions' two shuffles are shared by them. Only for pair
// kernels without a near field (the plane): a near verdict is not acted on here. A reaction
// would sum 32T terms in FP32 over the tile; it is restarted every 8 steps instead (8T terms, as
// many as the ordered FP32C kernel sums before promoting), and the four partials of a source,
// left in the lanes 8, 16, 24 and 32 places on, are added in FP64 into rud, rvd.
template <class V, int T>
__device__ __forceinline__ void react_tiles32_full(const f32::F32Geometry &f, const float4 (&t)[T],
                                                   const float (&tg)[T], const float4 *sf,
                                                   const float *sg, float (&u)[T], float (&v)[T],
                                                   double &rud, double &rvd) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
    float pu[4], pv[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        float ru = 0.0f, rv = 0.0f;
#pragma unroll 2
        for (int kk = 0; kk < 8; ++kk) {
            const int j = (lane + 8 * m + kk) & 31;
            const float4 s = sf[j];
            const float g = sg[j];
#pragma unroll
            for (int q = 0; q < T; ++q) {
                float ku, kv;
                V::values(f, t[q], s, ku, kv);
                u[q] = fmaf(-g, ku, u[q]);
                v[q] = fmaf(g, kv, v[q]);
                ru = fmaf(tg[q], ku, ru);
                rv = fmaf(-tg[q], kv, rv);
            }
            ru = __shfl_sync(0xffffffffu, ru, next);
            rv = __shfl_sync(0xffffffffu, rv, next);
        }
        pu[m] = ru;  // the partial of source (lane + 8 (m + 1)) & 31
        pv[m] = rv;
    }
    rud = static_cast<double>(__shfl_sync(0xffffffffu, pu[0], (lane - 8) & 31));
    rvd = static_cast<double>(__shfl_sync(0xffffffffu, pv[0], (lane - 8) & 31));
    rud += static_cast<double>(__shfl_sync(0xffffffffu, pu[1], (lane - 16) & 31));
    rvd += static_cast<double>(__shfl_sync(0xffffffffu, pv[1], (lane - 16) & 31));
    rud += static_cast<double>(__shfl_sync(0xffffffffu, pu[2], (lane - 24) & 31));
    rvd += static_cast<double>(__shfl_sync(0xffffffffu, pv[2], (lane - 24) & 31));
    rud += static_cast<double>(pu[3]);
    rvd += static_cast<double>(pv[3]);
}

template <class V = f32::Periodic32>
__device__ __forceinline__ void one_sided_tile32(const f32::F32Geometry &f, const float4 t,
                                                 bool t_ok, const float4 *sf, const float *sg,
                                                 int s_count, bool same_block, float &u,
                                                 float &v, const NearTile &nt) {
    const int lane = threadIdx.x & 31;
    for (int k = same_block ? 1 : 0; k < 32; ++k) {
        const int j = (lane + k) & 31;
        if (t_ok && j < s_count) {
            float ku, kv;
            if (V::values(f, t, sf[j], ku, kv))  // the other side lists its own pair
                list_near_pair<V>(nt, j, false);
            u = fmaf(-sg[j], ku, u);
            v = fmaf(sg[j], kv, v);
        }
    }
}

// (x_hi, y_hi, x_lo, y_lo) of a double position.
__device__ __forceinline__ float4 split32(double x, double y) { return f32::split_position(x, y); }

}  // namespace sym
}  // namespace pvb
