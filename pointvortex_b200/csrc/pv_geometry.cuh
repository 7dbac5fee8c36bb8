// pv_geometry.cuh — the three Biot–Savart pair interactions of PointVortex, FP64.
//
// Each geometry provides
//   * a per-source record staged in shared memory (x, y, and a scaled circulation),
//   * pair<CHECK>(): the fast form used by the tiled kernels, which adds one source's
//     contribution to one target's (u, v); CHECK enables the self-pair test and is only
//     instantiated for the diagonal tiles,
//   * slow_target(): the reference form with IEEE divisions and the reference's singular-pair
//     test, used to recompute a target whose fast-path sum came out non-finite. It returns the
//     reference's verdict (coincident pair / non-finite / finite).
#pragma once

#include "pv_common.cuh"

namespace pvb {

constexpr double kPi = 3.141592653589793;            // std::numbers::pi
constexpr double kInverseTwoPi = 0.5 / 3.141592653589793;

enum GeometryId : int { GEO_INFINITE = 0, GEO_PERIODIC = 1, GEO_DISK = 2 };

// Constants of one simulation, passed by value to every kernel (kernel parameter space).
struct GeometryConsts {
    int geometry;
    int image_layers;
    // infinite plane
    double eps2;            // coreRadius^2
    // periodic box (Weiss–McWilliams)
    double lx, ly;          // box lengths (square within 1e-13)
    double inv_lx, inv_ly;  // 1/L
    double half_lx, half_ly;
    double wave;            // 2 pi / Lx
    double half_wave;       // pi / Lx (exactly wave / 2)
    double scale;           // 0.5 / Lx
    int m_exact;            // image pairs m = +-1..m_exact summed exactly (min(M, 2))
    double cosh_m[3];       // cosh(2 pi m), m = 0..2
    double two_cosh_m[3];   // 2 cosh(2 pi m)
    double sinh2_m[3];      // sinh(2 pi m)^2
    double k1, k2;          // 2 sum sech(2 pi m), 2 sum sech^2(2 pi m) over m = 3..min(M, 6)
    // ZetaPair: the box's pair term as a rational function of z^4 (zeta != 0: it applies)
    int zeta;
    int half_hi;            // high word of L/2
    double zp[6], zq[3];    // numerator, and monic denominator of degree 3, in z^4
    double zs[8];           // box_energy: sigma(z)/z in z^4
    double energy_r2, energy_0;  // -pi/L^2 and the constant of the pair energy
    // disk
    double radius, radius2, inv_radius, inv_radius2;
    // FP32-compensated form: near-field radius squared (0: none), pv_pair32.cuh
    double near2;
};

// Scaled circulation stored per source, chosen so that each pair needs one multiply by it:
// infinite plane and disk Gamma/(2 pi) (the reference's inverseTwoPi * Gamma), periodic box
// Gamma * 0.5/L (the reference's scale * Gamma).
__host__ __device__ __forceinline__ double scaled_circulation(const GeometryConsts &g, double gamma) {
    if (g.geometry == GEO_PERIODIC)
        return g.scale * gamma;
    return kInverseTwoPi * gamma;
}

// ---------------------------------------------------------------------------------------------
// Infinite plane, src/compute.cpp:88-133: u -= (G/2pi) dy/(r^2+eps^2), v += (G/2pi) dx/(r^2+eps^2).
struct InfinitePair {
    template <bool CHECK>
    __device__ __forceinline__ static void pair(const GeometryConsts &g, double tx, double ty,
                                                double sx, double sy, double sg, bool self,
                                                double &u, double &v) {
        const double dx = tx - sx;
        const double dy = ty - sy;
        const double r2 = fma(dx, dx, fma(dy, dy, g.eps2));
        double c = sg * rcp_refined(r2);
        if (CHECK && self)
            c = 0.0;
        u = fma(-c, dy, u);
        v = fma(c, dx, v);
    }
};

// Disk of radius R, src/compute.cpp:286-336, with the source record of the infinite plane
// (x, y, G/(2 pi)). With p = z_i/R^2 and k = G/(2 pi):
//   direct (j != i):  u -= k dy/r^2,  v += k dx/r^2                 (dx = x_i - x_j, ...)
//   image (all j):    a = 1 - p.z_j, b = p_y x_j - p_x y_j,
//                     u += (k/R^2) (b x_j - a y_j)/(a^2 + b^2),  v += (k/R^2) (a x_j + b y_j)/(a^2 + b^2)
// which is the reference's circle-theorem image term written in unscaled source coordinates.
struct DiskPair {
    template <bool CHECK>
    __device__ __forceinline__ static void pair(const GeometryConsts &g, double tx, double ty,
                                                double sx, double sy, double sg, bool self,
                                                double &u, double &v) {
        const double dx = tx - sx;
        const double dy = ty - sy;
        const double r2 = fma(dx, dx, dy * dy);
        double c = sg * rcp_refined(r2);
        if (CHECK && self)
            c = 0.0;
        u = fma(-c, dy, u);
        v = fma(c, dx, v);
        image(g, tx, ty, sx, sy, sg, u, v);
    }
    // The direct term alone (j != i).
    __device__ __forceinline__ static void direct(double tx, double ty, double sx, double sy,
                                                  double sg, double &u, double &v) {
        const double dx = tx - sx;
        const double dy = ty - sy;
        const double c = sg * rcp_refined(fma(dx, dx, dy * dy));
        u = fma(-c, dy, u);
        v = fma(c, dx, v);
    }
    // The image term alone (every j, j == i included).
    __device__ __forceinline__ static void image(const GeometryConsts &g, double tx, double ty,
                                                 double sx, double sy, double sg, double &u,
                                                 double &v) {
        const double px = tx * g.inv_radius2, py = ty * g.inv_radius2;
        const double a = fma(-px, sx, fma(-py, sy, 1.0));
        const double b = fma(py, sx, -px * sy);
        const double ci = (sg * g.inv_radius2) * rcp_refined(fma(a, a, b * b));
        u = fma(ci, fma(b, sx, -a * sy), u);
        v = fma(ci, fma(a, sx, b * sy), v);
    }
};

// Periodic square box, src/compute.cpp:203-256 (Weiss–McWilliams image sum, truncated at
// |m| <= M with the reference's rule that an image whose |shift| exceeds 40 contributes 0).
//
// With x^ = (2 pi/L) remainder(dx, L), y^ likewise, the reference adds per source
//   u -= k sin(y^) sum_m 1/D_u(m),  D_u(m) = 2 (sinh^2((x^ - 2 pi m)/2) + sin^2(y^/2)),
//   v += k sin(x^) sum_m 1/D_v(m),  D_v(m) = 2 (sinh^2((y^ - 2 pi m)/2) + sin^2(x^/2)).
// The same truncated sum is evaluated here with one reciprocal per axis. With C = cosh x^,
// c = cos y^, a = 2 pi m, A = cosh a, D(m) = cosh(x^ - a) - c:
//   * m = 0 keeps the cancellation-free form 2 (sinh^2(x^/2) + sin^2(y^/2));
//   * m = +-1, +-2 (never dropped, since |x^| <= pi) combine exactly in pairs,
//       D(m) + D(-m) = 2 (C A - c),   D(m) D(-m) = C^2 + c^2 - 2 c C A + sinh^2 a,
//     where every term of the product is far from cancelling (sinh^2 a >= 7e4 > 2 |c| C A);
//   * m = +-3..+-6: with u = sech a <= 1.3e-8 the pair sum is
//       2u C + 2u^2 c cosh 2x^ + O(u^3 C^3),
//     and the omitted terms are below 1e-19 of the m = 0 term, far under FP64 rounding;
//   * the reference keeps an m = +-6 image only where |x^ -+ 12 pi| <= 40, so for |x^| > 2.3 it
//     drops one of the pair: a term of at most 2 e^{-12 pi} e^{-2.3} ~ 9e-18, below 1.2e-16 of the
//     sum (whose m = 0 part alone is at least 0.079). Both are kept here, which spares the
//     window test and sinh x^: the difference is at the level of the sum's own rounding;
//   * |m| >= 7 always has |shift| > 40 and is dropped, as in the reference.
// sinh, cosh, sin and cos of x^/2 and y^/2 come from one shared series (|x^/2| <= pi/2).
struct PeriodicPair {
    // Images m != 0 of one axis as num/den + rest: C = cosh of the axis, c = cos of the other.
    __device__ __forceinline__ static void image_sum(const GeometryConsts &g, double ch, double c,
                                                     double &num, double &den, double &rest) {
        const double ch2 = ch * ch;
        const double p = fma(c, c, ch2);   // C^2 + c^2
        const double m2c = -2.0 * c;
        const double q = m2c * ch;         // -2 c C
        // m = 1 starts the fraction, m = 2 joins it: num/den = pn1/pd1 + pn2/pd2
        num = 0.0;
        den = 1.0;
        if (g.m_exact >= 1) {
            num = fma(ch, g.two_cosh_m[1], m2c);
            den = fma(q, g.cosh_m[1], p + g.sinh2_m[1]);
        }
        if (g.m_exact >= 2) {
            const double pair_num = fma(ch, g.two_cosh_m[2], m2c);
            const double pair_den = fma(q, g.cosh_m[2], p + g.sinh2_m[2]);
            num = fma(pair_num, den, num * pair_den);
            den *= pair_den;
        }
        // m = 3..6: 2u C + 2u^2 c cosh 2x^ summed over u = sech(2 pi m), with
        // k2 cosh 2x^ = k2 (2 C^2 - 1) as one fma
        rest = fma(ch, g.k1, c * fma(2.0 * g.k2, ch2, -g.k2));
    }

    // The pair's terms without its circulation: the target's velocity changes by
    // u -= g_s * au / bu, v += g_s * av / bv. Exchanging target and source negates x^ and y^
    // exactly (remainder is odd), which negates au and av and leaves bu and bv unchanged, bit for
    // bit: every quantity below is an exactly odd or even function of (x^, y^).
    // HALF_SINE: au and av carry sin(y^)/2 and sin(x^)/2 (exactly half: the caller doubles the
    // circulation instead, which saves two multiplies per pair and changes no bit of the sums).
    template <bool HALF_SINE = false>
    __device__ __forceinline__ static void terms(const GeometryConsts &g, double tx, double ty,
                                                 double sx, double sy, double &au, double &bu,
                                                 double &av, double &bv) {
        // x^/2 and y^/2: pi/L times the remainder is exactly half of (2 pi/L) times it
        const double hx = g.half_wave * exact_remainder(tx - sx, g.lx, g.inv_lx, g.half_lx);
        const double hy = g.half_wave * exact_remainder(ty - sy, g.ly, g.inv_ly, g.half_ly);
        double shx, chx, snx, csx, shy, chy, sny, csy;
        sinh_cosh_sin_cos_economized(hx, shx, chx, snx, csx);
        sinh_cosh_sin_cos_economized(hy, shy, chy, sny, csy);
        const double tshx = 2.0 * shx, tshy = 2.0 * shy;    // scaling by 2 is exact
        const double nsnx = -2.0 * snx, nsny = -2.0 * sny;
        const double cosh_x = fma(tshx, shx, 1.0); // cosh x^ = 1 + 2 sinh^2(x^/2)
        const double cosh_y = fma(tshy, shy, 1.0);
        const double cos_x = fma(nsnx, snx, 1.0);  // cos x^ = 1 - 2 sin^2(x^/2)
        const double cos_y = fma(nsny, sny, 1.0);
        const double sin_x = HALF_SINE ? snx * csx : 2.0 * snx * csx; // sin x^ (or half)
        const double sin_y = HALF_SINE ? sny * csy : 2.0 * sny * csy;
        // 2 (sinh^2(x^/2) + sin^2(y^/2)) with the factor 2 inside: the same rounding, bit for bit
        const double d0u = fma(tshx, shx, -(nsny * sny));
        const double d0v = fma(tshy, shy, -(nsnx * snx));
        double nu, du, ru, nv, dv, rv;
        image_sum(g, cosh_x, cos_y, nu, du, ru);
        image_sum(g, cosh_y, cos_x, nv, dv, rv);
        // 1/d0 + num/den + rest = (den + d0 (num + den rest)) / (d0 den)
        au = sin_y * fma(d0u, fma(du, ru, nu), du);
        av = sin_x * fma(d0v, fma(dv, rv, nv), dv);
        bu = d0u * du;
        bv = d0v * dv;
    }

    template <bool CHECK>
    __device__ __forceinline__ static void pair(const GeometryConsts &g, double tx, double ty,
                                                double sx, double sy, double sg, bool self,
                                                double &u, double &v) {
        if (CHECK && self) // the self pair contributes exactly 0 in the reference (sin 0 = 0)
            return;
        double au, bu, av, bv;
        terms(g, tx, ty, sx, sy, au, bu, av, bv);
        u = fma(-(sg * au), rcp_refined(bu), u);
        v = fma(sg * av, rcp_refined(bv), v);
    }
};

// The same box from six images up, as one rational function of the complex displacement.
//
// With z = x + iy the reduced displacement, W = K_v - i K_u (the pair changes its target by
// u -= g K_u, v += g K_v) is the doubly periodic velocity of a vortex and its images,
//   W(z) = (L/pi) [ zeta(z) - pi conj(z)/L^2 ],
// zeta being Weierstrass' zeta function of the lattice L, iL: both image sums of the reference
// (x-images for u, y-images for v) converge to its parts. Its truncations are there below rounding
// from M = 6: a dropped image |m| >= 7 is below e^{-13 pi} ~ 2e-18 of the sum, and the reference's
// own cut drops one of m = +-6 (PeriodicPair's comment: below 1.2e-16 of the sum).
//
// On a square lattice zeta(iz) = -i zeta(z), so z zeta(z) is a function of z^4 alone, analytic but
// for real poles at z^4 = L^4 and beyond. Over the box |x|, |y| <= L/2 it equals
//   z zeta(z) = P(z^4) / Q(z^4),  P of degree 5, Q of degree 3, real coefficients,
// within 6.6e-18 (weighted least squares on the boundary of the box, iterated to equal ripple, 50
// digits; the maximum principle bounds the interior). P and Q at a complex argument take two real
// operations a degree (Knuth's recurrence in 2 Re w and |w|^2), and one reciprocal of |z Q|^2
// serves both components: 50 FP64 instructions for an unordered pair where PeriodicPair needs 119
// (its two half-angle series alone 44). Evaluated in FP64 the term is within 6e-16 of itself
// everywhere in the box (PeriodicPair: 4e-15), close pairs included: x and y enter as they are.
// Exchanging the vortices negates x and y, which leaves w, P and Q and negates the terms, exactly.
//
// What bounds it is the FP64 pipe: two cycles an instruction, three where all operands are distinct
// registers (17 of the 50). Measured per evaluation inside DOPRI5 steps (B200), PeriodicPair against
// this: N = 2048 43 -> 26 us, 4096 84 -> 46 us, 16 384 1084 -> 495 us, 65 536 17.2 -> 7.55 ms; the
// ordered kernel at N = 16 384 2170 -> 1048 us.
constexpr int kZetaMinLayers = 6;
// L^25 and its reciprocal have to stay normal numbers: other boxes keep PeriodicPair.
constexpr double kZetaMinLength = 1.0 / 65536.0, kZetaMaxLength = 65536.0;
// Coefficients for L = 2 (z^4 in [-4, 1] on the real axis); the host scales them to the box.
constexpr double kZetaP[6] = {0.99999999999999999987, -0.24693625978040467126,
                              -0.0076101740589869094825, 3.5984216120403640632e-05,
                              5.3640689704854244344e-09, 2.566617850026110922e-10};
constexpr double kZetaQ[4] = {1.0, -0.04998550964578607478, -0.00083074426019041809798,
                              3.0367890005030402872e-06};

// The same function in units of L/2 with a monic denominator: kZetaP (2/pi) / kZetaQ[3] and
// kZetaQ / kZetaQ[3]. With these the coefficients are literals (UNIT below).
__host__ __device__ constexpr double zeta_unit_p(int k) {
    return k == 0   ? 2.0963582661229544646e+5
           : k == 1 ? -5.1766686939613659311e+4
           : k == 2 ? -1.5953651295191684159e+3
           : k == 3 ? 7.5435808913963043333
           : k == 4 ? 1.1245010326330765775e-3
                    : 5.3805505458809630715e-5;
}
__host__ __device__ constexpr double zeta_unit_q(int k) {
    return k == 0   ? 3.2929518640720552362e+5
           : k == 1 ? -1.6459987716468295239e+4
                    : -2.7356008601611977445e+2;
}

// sigma(z)/z as a polynomial in z^4 over the box (relative error 8.8e-19, fitted as kZetaP), and the
// constant of box_energy in units of the reduced displacement (2 pi/L) z.
constexpr double kZetaS[8] = {1.0, -4.9237687533654649034e-2, -8.6583924059350373423e-4,
                              2.2856275188869999334e-6, 1.0998971914462181745e-9,
                              2.2669498722569394859e-11, 3.886542270771162172e-15,
                              -1.1103889041850561031e-17};
constexpr double kEnergyConstant = -0.7006448850558935816776;

// 2 v and 4 v by the exponent, off the FP64 pipe. A zero becomes about 1e-308, which no sum below
// can see; no infinity reaches this, and a NaN also enters the term through |w|^2.
__device__ __forceinline__ double exponent_up(double v, int powers) {
    return __hiloint2double(__double2hiint(v) + (powers << 20), __double2loint(v));
}

// UNIT: the coefficients as literals for displacements in units of L/2, at two multiplications a
// pair. For kernels whose GeometryConsts is not a kernel parameter (the ensembles': one box after
// another), where each coefficient would be a load from shared memory for every pair.
template <bool UNIT> struct ZetaPairT {
    // The kernel values of a reduced displacement.
    __device__ __forceinline__ static void terms(const GeometryConsts &g, double x, double y,
                                                 double &ku, double &kv) {
        double zp[6], zq[3];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            zp[k] = UNIT ? zeta_unit_p(k) : g.zp[k];
            if (k < 3)
                zq[k] = UNIT ? zeta_unit_q(k) : g.zq[k];
        }
        if (UNIT) {
            x *= 2.0 * g.inv_lx;
            y *= 2.0 * g.inv_lx;
        }
        const double linear = UNIT ? 0.5 : g.inv_lx;
        const double yy = y * y;
        const double a = fma(x, x, -yy), r = fma(x, x, yy), b = x * y;  // z^2 = a + 2ib, r = |z|^2
        const double r2 = r * r, n = r2 * r2;                           // |w|^2, w = z^4
        const double wr = fma(-8.0 * b, b, r2);
        const double wi = exponent_up(a * b, 2);
        const double tr = exponent_up(wr, 1);
        const double p4 = fma(tr, zp[5], zp[4]);
        const double p3 = fma(tr, p4, fma(-n, zp[5], zp[3]));
        const double p2 = fma(tr, p3, fma(-n, p4, zp[2]));
        const double p1 = fma(tr, p2, fma(-n, p3, zp[1]));
        const double pr = fma(wr, p1, fma(-n, p2, zp[0])), pi = wi * p1;
        const double q2 = tr + zq[2];
        const double q1 = fma(tr, q2, zq[1] - n);
        const double qr = fma(wr, q1, fma(-n, q2, zq[0])), qi = wi * q1;
        const double dr = fma(x, qr, -y * qi), di = fma(x, qi, y * qr);  // z Q
        const double inv = rcp_refined(fma(dr, dr, di * di));
        ku = fma(fma(pr, di, -pi * dr), inv, -linear * y);
        kv = fma(fma(pr, dr, pi * di), inv, -linear * x);
    }

    // remainder(d, L) for |d| <= 3L/2: one subtraction of 0 or +-L (exact, as the remainder is),
    // chosen on the integer pipe. At the seam |x| may pass L/2 by 2^-20 of it, where the term is
    // as good.
    __device__ __forceinline__ static double reduce_near(const GeometryConsts &g, double d,
                                                         double length) {
        const int hi = __double2hiint(d);
        const bool far = (hi & 0x7fffffff) > g.half_hi;
        const double shift = __hiloint2double(
            far ? (__double2hiint(length) | (hi & static_cast<int>(0x80000000u))) : 0,
            far ? __double2loint(length) : 0);
        return d - shift;
    }
    // Whether reduce_near() serves every difference of such coordinates.
    __device__ __forceinline__ static bool inside(const GeometryConsts &g, double x, double y) {
        return fabs(x) <= 1.5 * g.half_lx && fabs(y) <= 1.5 * g.half_ly;
    }

    // remainder(a, L) of any difference: the nearest multiple by adding and taking off 1.5 2^52, and
    // NaN for what that cannot reach (beyond 2^51 boxes), which sends the target to the reference
    // form's recomputation. The test is on the integer pipe and leaves no branch in a pair loop
    // (with a call of the library's remainder there, a loop's pairs ran one after another: 17 800
    // cycles against 5800 for a chunk of 34 sources in the cooperative steps at N = 1024).
    __device__ __forceinline__ static double reduce(const GeometryConsts &g, double a,
                                                    double length, double inv_length) {
        const double n = __dadd_rn(fma(a, inv_length, 6755399441055744.0), -6755399441055744.0);
        const double r = fma(-n, length, a);
        const int hi = __double2hiint(r);
        return __hiloint2double((hi & 0x7fffffff) > g.half_hi ? 0x7ff80000 : hi, __double2loint(r));
    }
    // The same with the library's remainder instead of NaN.
    __device__ __forceinline__ static double reduce_any(const GeometryConsts &g, double a,
                                                        double length, double inv_length) {
        const double n = __dadd_rn(fma(a, inv_length, 6755399441055744.0), -6755399441055744.0);
        const double r = fma(-n, length, a);
        if ((__double2hiint(r) & 0x7fffffff) > g.half_hi)
            return remainder(a, length);
        return r;
    }

    template <bool CHECK>
    __device__ __forceinline__ static void pair(const GeometryConsts &g, double tx, double ty,
                                                double sx, double sy, double sg, bool self,
                                                double &u, double &v) {
        double ku, kv;
        terms(g, reduce(g, tx - sx, g.lx, g.inv_lx), reduce(g, ty - sy, g.ly, g.inv_ly), ku, kv);
        if (CHECK && self)  // contributes exactly 0 in the reference
            ku = kv = 0.0;
        u = fma(-sg, ku, u);
        v = fma(sg, kv, v);
    }
};
using ZetaPair = ZetaPairT<false>;
using ZetaUnitPair = ZetaPairT<true>;

// One ordered pair of the box, by the form its constants allow.
template <bool CHECK>
__device__ __forceinline__ void periodic_pair(const GeometryConsts &g, double tx, double ty,
                                              double sx, double sy, double sg, bool self, double &u,
                                              double &v) {
    if (g.zeta)
        ZetaPair::pair<CHECK>(g, tx, ty, sx, sy, sg, self, u, v);
    else
        PeriodicPair::pair<CHECK>(g, tx, ty, sx, sy, sg, self, u, v);
}

// The box's pair energy in the same units, -x^2/(2 pi) + sum_m [log D(m) - log cosh(2 pi m)] of the
// reference (x, y here times 2 pi/L), which is 2 log|sigma(z)| - pi |z|^2/L^2 + constant: sigma is
// entire, sigma(z)/z a function of z^4 alone, and a polynomial of degree 7 over the box. One logarithm
// a pair, of the argument |z|^2 |S|^2 (0 only for z = 0), added to `rest`, and 30 more FP64
// instructions; the image product it replaces took two logarithms, both half-angle series and four
// instructions an image.
__device__ __forceinline__ double box_energy(const GeometryConsts &g, double x, double y,
                                             double &rest) {
    const double yy = y * y;
    const double a = fma(x, x, -yy), r = fma(x, x, yy), b = x * y;
    const double r2 = r * r, n = r2 * r2;
    const double wr = fma(-8.0 * b, b, r2);
    const double wi = exponent_up(a * b, 2);
    const double tr = exponent_up(wr, 1);
    double s2 = g.zs[7], s1 = fma(tr, s2, g.zs[6]);  // Knuth's recurrence downwards
#pragma unroll
    for (int k = 5; k >= 1; --k) {
        const double s0 = fma(tr, s1, fma(-n, s2, g.zs[k]));
        s2 = s1;
        s1 = s0;
    }
    const double sr = fma(wr, s1, fma(-n, s2, g.zs[0])), si = wi * s1;
    rest = fma(r, g.energy_r2, g.energy_0);
    return r * fma(sr, sr, si * si);
}

// ---------------------------------------------------------------------------------------------
// Reference-form recomputation of one target (IEEE divisions, library sinh/sin/remainder,
// the reference's singular-pair rule). Verdict: 0 finite, ST_COINCIDENT, ST_NONFINITE_VELOCITY.
__device__ inline int slow_target(const GeometryConsts &g, const double *x, const double *y,
                                  const double *gamma, size_t n, size_t t, double &u_out,
                                  double &v_out) {
    double u = 0.0, v = 0.0;
    int singular = 0;
    const double tx = x[t], ty = y[t];
    if (g.geometry == GEO_INFINITE) {
        for (size_t s = 0; s < n; ++s) {
            if (s == t)
                continue;
            const double dx = tx - x[s], dy = ty - y[s];
            const double den = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), g.eps2);
            if (den == 0.0) {
                singular = 1;
                continue;
            }
            const double c = __dmul_rn(kInverseTwoPi, gamma[s]) / den;
            u -= c * dy;
            v += c * dx;
        }
    } else if (g.geometry == GEO_PERIODIC) {
        const int layers = g.image_layers;
        for (size_t s = 0; s < n; ++s) {
            const double sdx = g.wave * remainder(tx - x[s], g.lx);
            const double sdy = g.wave * remainder(ty - y[s], g.ly);
            const double sine_x = sin(sdx), sine_y = sin(sdy);
            const double shx = sin(0.5 * sdx), shy = sin(0.5 * sdy);
            for (int m = -layers; m <= layers; ++m) {
                if (s == t && m == 0)
                    continue;
                const double shift = __dmul_rn(2.0 * kPi, static_cast<double>(m));
                const double ax = __dsub_rn(sdx, shift), ay = __dsub_rn(sdy, shift);
                double du, dv;
                if (fabs(ax) > 40.0) {
                    du = __longlong_as_double(0x7ff0000000000000ll);
                } else {
                    const double h = sinh(0.5 * ax);
                    du = 2.0 * __dadd_rn(__dmul_rn(h, h), __dmul_rn(shy, shy));
                }
                if (fabs(ay) > 40.0) {
                    dv = __longlong_as_double(0x7ff0000000000000ll);
                } else {
                    const double h = sinh(0.5 * ay);
                    dv = 2.0 * __dadd_rn(__dmul_rn(h, h), __dmul_rn(shx, shx));
                }
                if (du == 0.0 || dv == 0.0) {
                    singular = 1;
                    continue;
                }
                u -= __dmul_rn(__dmul_rn(g.scale, gamma[s]), sine_y) / du;
                v += __dmul_rn(__dmul_rn(g.scale, gamma[s]), sine_x) / dv;
            }
        }
    } else {
        const double ir = g.inv_radius;
        const double txs = tx * ir, tys = ty * ir;
        for (size_t s = 0; s < n; ++s) {
            if (s != t) {
                const double dx = tx - x[s], dy = ty - y[s];
                const double den = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
                if (den == 0.0) {
                    singular = 1;
                    continue;
                }
                const double c = __dmul_rn(kInverseTwoPi, gamma[s]) / den;
                u -= c * dy;
                v += c * dx;
            }
            const double sx = x[s] * ir, sy = y[s] * ir;
            const double a = 1.0 - __dadd_rn(__dmul_rn(txs, sx), __dmul_rn(tys, sy));
            const double b = __dsub_rn(__dmul_rn(tys, sx), __dmul_rn(txs, sy));
            const double den = __dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b));
            const double ix = __dsub_rn(__dmul_rn(-a, sx), __dmul_rn(b, sy));
            const double iy = __dadd_rn(__dmul_rn(-a, sy), __dmul_rn(b, sx));
            const double c = __dmul_rn(__dmul_rn(-kInverseTwoPi, gamma[s]), ir) / den;
            u -= c * iy;
            v += c * ix;
        }
    }
    u_out = u;
    v_out = v;
    if (singular)
        return ST_COINCIDENT;
    if (!isfinite(u) || !isfinite(v))
        return ST_NONFINITE_VELOCITY;
    return 0;
}

} // namespace pvb
