// FP64 filter of the lane-packing criteria: the verdict of a box from one
// round-to-nearest evaluation and an error bound, instead of two directed
// roundings of every step.
//
// filter_box evaluates the quantities that the criteria of a family compare
// (the same interval ends, combined by the same formulas, cp_families.cuh) in
// round-to-nearest FP64 and decides each comparison only when its two sides are
// further apart than the error bound.  Where every comparison on the way to the
// verdict is decided, the verdict is the one of eval_box; any other box is left
// to eval_box, bit for bit as before.
//
// Error bound.  "Directed" is eval_box's value, "filter" the value here, both
// against the same formula in exact arithmetic.  The box guard (box_ok) bounds
// the inputs: lambda in [kLambdaLow, kLambdaHigh], radii at most kMaxRadius, so that
// 0.25 <= L, S < 1.4.
//   * Directed: L^2 - S^2 and (a + b)^2 are off by at most 2^-49.4 (a few ulps of
//     values below 2), the quotient q = (L^2 - S^2 +- c^2) / (2 c L) of a
//     collision angle by 2^-49.4 / c <= 2^-41.4 (c = a + b >= 2^-8), and asin(q) by
//     2^-41.4 / sqrt(2 (1 - |q|)) <= 2^-33.9 where 1 - |q| >= kEnd = 2^-16.  Its
//     padding of asin (5 ulps) is far below that.
//   * Filter: the numerators carry the same roundings; the reciprocal is off by
//     at most 2^-38 of its value (a 2^-19 seed, checked over all its seeds in
//     tests/test_filter_gpu.py, and one Newton step); 1 - |q| is formed from the
//     numerators, not from q, so that its relative error stays small near 1; the
//     arcsine polynomial is off by 1e-12 of its value (2^-39.9).
// Every comparison sums at most three collision angles and three semicircle
// angles: both sides stay within 2^-31 of the exact formula, and kTau = 2^-30
// separates them.  (Angles enter the area comparisons with a factor of at most
// 1 - lambda^2, and so does the bound.)
//
// Trap sites and clamps.  eval_box's trap sites are domain and emptiness tests of
// the quotients.  Each corner that eval_box could evaluate is certified here to
// stay clear of them (the comments at the corners say why); where it is not, the
// box is left to eval_box.
//
// What it gives: the directed evaluation is bound by issue and by the latency of
// about 24 certified divisions and 12 padded arcsines per box, each a call.  Here
// a collision angle costs one approximate reciprocal and two short polynomials,
// inlined, and most boxes are decided from a few of their angles.  About 1 in 5000
// lattice boxes is left to eval_box.  On B200: 1e6 complete masks (middle) 388 -> 93 us.
// What it gave refinements by itself, while every box still passed through a level: 64^4
// middle lattice and two uniform levels 494 -> 188 ms, half of the start proof 74.6 ->
// 33.8 ms (they take 76 and 26 ms now, cp_refine.cuh).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CPF_HD __host__ __device__ __forceinline__
#else
#define CPF_HD inline
#endif
#include <cmath>

namespace cpb {
namespace flt {

// What the caller consumes of a decided box.
enum Need : int {
    NEED_VERDICT = 0,  // the verdict alone
    NEED_HANDLES = 1,  // the verdict and the number of guarded criteria evaluated (DECIDE order)
    NEED_MASK = 2,     // the fail mask of DECIDE order
    NEED_FULL = 3      // the complete fail mask
};

constexpr double kTau = 9.313225746154785e-10;   // 2^-30, bound on an angle sum's error
constexpr double kAbs = 1.4210854715202004e-14;  // 2^-46, bound on the area terms' own roundings
constexpr double kEnd = 1.52587890625e-05;       // 2^-16, least distance of a quotient from 1
constexpr double kTie = 1.4210854715202004e-14;  // 2^-46, least distance from the obtuse/acute boundary
constexpr double kGap = 9.313225746154785e-10;   // 2^-30, least excess of 2 (a + b) over the lane width
constexpr double kMinB = 0.000244140625;             // 2^-12
constexpr double kLowSlack = 3.814697265625e-06;     // 2^-18
constexpr double kMinC = 0.00390625;                // 2^-8, least a + b
constexpr double kLambdaLow = 0.49, kLambdaHigh = 0.992, kMaxRadius = 0.3333;
constexpr double kHalfPi = 1.5707963267948966;
constexpr double kRatio = 0.5642, kPi = 3.141592653589793;  // lane_packing/values.hpp:28-32

// ------------------------------------------------------------------ arithmetic
CPF_HD double fma_(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
CPF_HD double abs_(double x) { return fabs(x); }
// seeds of 1/d and 1/sqrt(d): the FP64 approximations, within 2^-19 (host: rounded to
// float, or off by the relative error CPF_SEED_ERROR)
CPF_HD double rcp_seed_(double d) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return y;
#elif defined(CPF_SEED_ERROR)
    return (1.0 + (CPF_SEED_ERROR)) / d;
#else
    return (double)(1.0f / (float)d);
#endif
}
CPF_HD double rsqrt_seed_(double d) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return y;
#elif defined(CPF_SEED_ERROR)
    return (1.0 + (CPF_SEED_ERROR)) / std::sqrt(d);
#else
    return (double)(1.0f / std::sqrt((float)d));
#endif
}
CPF_HD double rcp_(double d) {
    const double y = rcp_seed_(d);
    return fma_(y, fma_(-d, y, 1.0), y);
}
CPF_HD double rsqrt_(double d) {
    const double y = rsqrt_seed_(d);
    return fma_(0.5 * y, fma_(-d * y, y, 1.0), y);
}
// RD(x + y) and RU(x + y), for the comparisons that are exact
CPF_HD double add_rd_(double x, double y) {
#ifdef __CUDA_ARCH__
    return __dadd_rd(x, y);
#else
    const double s = x + y, t = s - x;
    return (x - (s - t)) + (y - t) < 0.0 ? std::nextafter(s, -4.0) : s;
#endif
}
CPF_HD double add_ru_(double x, double y) { return -add_rd_(-x, -y); }
CPF_HD double mul_rd_(double x, double y) {
#ifdef __CUDA_ARCH__
    return __dmul_rd(x, y);
#else
    const double p = x * y;
    return fma_(x, y, -p) < 0.0 ? std::nextafter(p, -4.0) : p;
#endif
}
CPF_HD double mul_ru_(double x, double y) { return -mul_rd_(-x, y); }
// the next double above a positive x
CPF_HD double above_(double x) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(__double_as_longlong(x) + 1);
#else
    return std::nextafter(x, 1e300);
#endif
}

// asin(x) = x + x z P(z), z = x^2, |x| <= 1/2: minimax polynomial (Remez exchange
// on z in [0, 1/4], relative error 9.8e-13).
CPF_HD double asin_core(double x, double z) {
    double p = 0.03289646763320449;
    p = fma_(p, z, 0.0019933684297839347);
    p = fma_(p, z, 0.020640993408479382);
    p = fma_(p, z, 0.02186676674568419);
    p = fma_(p, z, 0.030426411564165902);
    p = fma_(p, z, 0.044640714121541566);
    p = fma_(p, z, 0.07500004965298718);
    p = fma_(p, z, 0.16666666627480178);
    return fma_(x * z, p, x);
}
// asin(n / d) for |n| <= d, r = 1/d: beyond 1/2 from 1 - |n|/d = (d - |n|) r.
// ok: the quotient keeps kEnd away from 1.  One polynomial for both ranges, so that
// lanes on either side of 1/2 share it.
CPF_HD double asin_pos(double n, double d, double r, bool& ok) {
    const double x = n * r;
    const bool far = n + n > d;
    double s = x, z = x * x;
    if (far) {
        z = (0.5 * r) * (d - n);
        ok = ok && z >= 0.5 * kEnd;
        s = z * rsqrt_(z);
    }
    const double p = asin_core(s, z);
    return far ? fma_(-2.0, p, kHalfPi) : p;
}
CPF_HD double asin_quot(double n, double d, double r, bool& ok) {
    return copysign(asin_pos(abs_(n), d, r, ok), n);
}

// ------------------------------------------------------------------ collision angles
// Disks of radii ro (touching the outer border, centre distance P = 1 - ro) and
// ri (touching the inner one, Q = lambda + ri, an interval [ql, qh] through lambda),
// upper corner, c = ro + ri.  The longer side is L = P, the shorter S = Q; where P
// lies below qh the reference takes the other order too (collision_angles.cu:144-158),
// the radii then nearly add up to the lane width: about 1 in 500 boxes of a coarse
// lattice, fewer of a finer one, left to eval_box.
// The wanted bound is asin((P^2 - ql^2 + c^2) / (2 c P)) minus asin((P^2 - qh^2 - c^2)
// / (2 c S)), S = qh where the angle at S is obtuse, else ql: the obtuse and acute
// formulas (collision_angles.cu:59-117) agree at their boundary, so a comparison near
// it needs no care.
// Trap sites: the first quotient exceeds 1 only when 2 c <= 1 - lambda.lo (to
// rounding), where the directed value is clamped if the angle is definitely obtuse
// and a trap otherwise.  The second exceeds 1 only beyond qh + c < P.
CPF_HD double mixed_hi(double ll, double lh, double ro, double ri, bool& ok) {
    const double P = 1.0 - ro, ql = ll + ri, qh = lh + ri, c = ro + ri;
    const double c2 = c * c, cc = c + c, P2 = P * P;
    const double n1 = fma_(-ql, ql, P2 + c2), n2 = fma_(-qh, qh, P2 - c2);
    const double d1 = cc * P, d2 = cc * (n2 > 0.0 ? qh : ql);
    const double r = rcp_(d1 * d2);
    ok = ok && qh <= P;
    double v1;
    if (n1 > d1) {  // clamped to 1: definitely obtuse, clear of 1, lower quotient inside
        ok = ok && n2 > kTie && n1 - d1 >= kEnd * d1 && d1 - (n2 + 2.0 * c2) >= kEnd * d1;
        v1 = kHalfPi;
    } else {
        v1 = asin_pos(n1, d1, r * d2, ok);
    }
    return v1 - asin_quot(n2, d2, r * d1, ok);
}
// the exact test of collision_angles.cu:160-173: disks that possibly fit side by side
CPF_HD bool side_by_side(double ll, double ro, double ri) { return 2.0 * add_rd_(ro, ri) <= add_ru_(1.0, -ll); }
// Lower corner: 0 side by side, else asin((P^2 - qh^2 + c^2) / (2 c P)) minus
// asin((P^2 - ql^2 - c^2) / (2 c S)) (S = ql where possibly obtuse, else qh), at
// least 0; the second quotient is clamped to 1.
// Trap sites: unless definitely obtuse, (P^2 - ql^2 + c^2) / (2 c P) > 1; if obtuse,
// (P^2 - qh^2 - c^2) / (2 c qh) > 1.
CPF_HD double mixed_lo(double ll, double lh, double ro, double ri, bool& ok) {
    if (side_by_side(ll, ro, ri)) return 0.0;
    const double P = 1.0 - ro, ql = ll + ri, qh = lh + ri, c = ro + ri;
    const double c2 = c * c, cc = c + c, P2 = P * P;
    const double n1 = fma_(-qh, qh, P2 + c2), n2 = fma_(-ql, ql, P2 - c2);
    const double d1 = cc * P, d2 = cc * (n2 > 0.0 ? ql : qh);
    const double r = rcp_(d1 * d2);
    const double al = n1 - c2;  // P^2 - qh^2
    if (al <= c2 + kTie) {
        ok = ok && qh <= P && d1 - (n2 + 2.0 * c2) >= kEnd * d1;
    } else {
        const double d3 = cc * qh;
        ok = ok && qh <= P && d3 - (al - c2) >= kEnd * d3;
    }
    double v2;
    if (n2 > d2) {
        ok = ok && n2 - d2 >= kEnd * d2;
        v2 = kHalfPi;
    } else {
        v2 = asin_quot(n2, d2, r * d1, ok);
    }
    const double v = asin_pos(n1, d1, r * d2, ok) - v2;
    return v < 0.0 ? 0.0 : v;
}
// Certificates for corners whose value is not needed.  They hold for either order of
// P and Q: with D = 2 (a + b) - (1 - lambda.lo) > 0 no quotient of a mixed corner
// exceeds 1, in the order L = P the excess is -D (P - c + ql), in the order L = Q it
// is bounded by the box guard.
// Below that, a definitely obtuse corner tests the lower ends of its quotients only.
// end_3d's radius ranges end where those are 1 to the last bit, so no margin can
// decide it: the directed chain itself is followed, the quotient add.lo = RD(num / ch)
// compared by multiplication.  RD(add.lo + cl) / 2 exceeds L.hi, by the reference's
// test RD(. / L.hi) > 1 as well as by emptiness, when add.lo + cl >= the double above
// 2 L.hi; RD(add.lo - ch) / 2 exceeds S.hi likewise.
CPF_HD bool clear_mixed_hi(double ll, double lh, double ro, double ri) {
    const double c = ro + ri;
    bool clear = 2.0 * c - (1.0 - ll) >= kGap;
    if (!clear) {
        const double P = 1.0 - ro, qh = lh + ri;
        const double cl = add_rd_(ro, ri), ch = add_ru_(ro, ri);
        const double l_lo = add_rd_(1.0, -ro), l_hi = add_ru_(1.0, -ro), s_hi = add_ru_(lh, ri);
        const double num = add_rd_(mul_rd_(l_lo, l_lo), -mul_ru_(s_hi, s_hi));
        clear = qh < P && fma_(P, P, -(qh * qh)) - c * c > kTie &&
                num < mul_rd_(add_rd_(above_(2.0 * l_hi), -cl), ch) &&
                num < mul_rd_(add_rd_(above_(2.0 * s_hi), ch), ch);
    }
    return clear;
}
CPF_HD bool clear_mixed_lo(double ll, double ro, double ri) {
    return side_by_side(ll, ro, ri) || 2.0 * (ro + ri) - (1.0 - ll) >= kGap;
}

// Two disks on the same border, a >= b: near-point sides L = x + a, S = x + b
// (inner, x = lambda) or 1 - b, 1 - a (outer), twox + c = L + S, so the angle is
// the point formula cos = 1 - 2 a b / (L S): 2 asin(sqrt(a b / (L S))).  1 - q >=
// b / c keeps the directed evaluation clear of 1 for b >= kMinB, and |L^2 - S^2 -
// c^2| > kTie clear of an empty partial result at the obtuse/acute boundary.
CPF_HD double excess(double a, double b, double sides) {
    const double c = a + b;
    return fma_(a - b, sides, -(c * c));  // L^2 - S^2 - c^2
}
CPF_HD bool clear_same(double a, double b, double sides) {
    return a >= b && b >= kMinB && abs_(excess(a, b, sides)) > kTie;
}
// Lower corner of a radius b below kMinB (end_3d: down to 0): definitely obtuse, both
// quotients at most 1 before their rounding, which is downward, so no trap site is
// reached; the directed value lies within kLowSlack below the angle.
CPF_HD bool clear_same_low(double a, double b, double sides) {
    return a >= b && (b >= kMinB ? abs_(excess(a, b, sides)) > kTie : excess(a, b, sides) > kTie);
}
CPF_HD double sides_inner(double x, double a, double b) { return 2.0 * x + (a + b); }
CPF_HD double sides_outer(double a, double b) { return 2.0 - (a + b); }
CPF_HD double same_angle(double a, double b, double L, double S) {
    double ab = a * b;
    if (ab < 1e-30) ab = 1e-30;  // b = 0: an angle of 2e-15
    const double s = ab * rsqrt_(ab * (L * S));
    return 2.0 * asin_core(s, s * s);
}
CPF_HD double inner_angle(double x, double a, double b) { return same_angle(a, b, x + a, x + b); }
CPF_HD double outer_angle(double a, double b) { return same_angle(a, b, 1.0 - a, 1.0 - b); }

// collision_angles.cu:233-246, quotients at most 1/2
CPF_HD double semi_angle(double r, double d) {
    const double x = r * rcp_(d);
    return asin_core(x, x * x);
}
CPF_HD double semi_outer(double r) { return semi_angle(r, 1.0 - r); }
CPF_HD double semi_inner(double x, double r) { return semi_angle(r, x + r); }

// x < y, decided only when they are more than tol apart
CPF_HD bool less_(double x, double y, double tol, bool& ok) {
    const double d = y - x;
    ok = ok && abs_(d) > tol;
    return d > 0.0;
}

// ------------------------------------------------------------------ boxes
struct FBox {
    double ll, lh;             // lambda
    double l1, h1, l2, h2, l3, h3;  // radii (lower ends tightened)
};
// The guard of the error bound (negated comparisons, so NaN fails): see the file
// comment.  lh - ll >= 2^-40 keeps the two ends of a mixed corner's L^2 - S^2 apart,
// so that they do not both fall on the obtuse/acute boundary; the last test bounds
// the first quotient of the order L = Q: (1 - lh)(P + qh - c) > 2 c (lh - ll).
template <bool THREE>
CPF_HD bool box_ok(const FBox& b) {
    const double w = b.lh - b.ll;
    double m = b.h1 > b.h2 ? b.h1 : b.h2;
    bool ok = b.ll >= kLambdaLow && b.lh <= kLambdaHigh && w >= 9.094947017729282e-13;
    ok = ok && b.l1 > 0.0 && b.l2 >= 0.0 && b.l1 <= b.h1 && b.l2 <= b.h2 && b.h1 + b.h2 >= kMinC;
    if (THREE) {
        ok = ok && b.l3 >= 0.0 && b.l3 <= b.h3 && b.h2 + b.h3 >= kMinC && b.l1 + b.l3 >= 0.5 * kMinC;
        if (b.h3 > m) m = b.h3;
    }
    ok = ok && m <= kMaxRadius;
    return ok && (1.0 - b.lh) * (1.0 + b.lh - 2.0 * m) >= fma_(4.0 * m, w, kGap);
}

// Where a box comes from: load() gives it with its radii tightened.  On the device it
// reads memory again each time (ref.load() is opaque to the compiler), so that no
// stage of an evaluation holds the box, or terms it shares with another stage, in
// registers: with all stages inlined and sharing, the kernels spilled 600 B a thread.
struct ValRef {  // a box in registers
    FBox b;
    CPF_HD FBox load() const { return b; }
};
CPF_HD void tighten(FBox& b, bool three) {
    if (three && b.l2 < b.l3) b.l2 = b.l3;
    if (b.l1 < b.l2) b.l1 = b.l2;
}

struct Terms {
    double ratio, tol;
    CPF_HD explicit Terms(const FBox& b) : ratio(fma_(-b.ll, b.ll, 1.0)), tol(fma_(kTau, ratio, kAbs)) {}
};
CPF_HD double disk_area(double l) { return kPi * (l * l); }

struct FOut {
    uint8_t mask;     // NEED_MASK / NEED_FULL: failing sub-criteria; else nonzero when a criterion fails
    uint8_t handles;  // NEED_HANDLES
};

// middle_configuration.cu:86-154.  The handle fails when (g1 and A) or (g2 and B):
// g1, g2 its two guards, A, B its two area tests.  c13.hi <= (c12 + c23).lo rules
// out c13.lo > (c12 + c23).hi (directed bounds of angles that grow with the
// radii), so g1 or g2 always holds: a handle whose tests both fail (both hold)
// fails (holds) whatever its guards say, and they are evaluated only in between.
template <int NEED, bool INNER, class Ref>
CPF_HD uint8_t middle_handle(const Ref& ref, bool& ok) {
    bool fa, fb;
    double c12_hi, c13_hi;
    {
        const FBox b = ref.load();
        const Terms t(b);
        const double k = 0.5 * kRatio * t.ratio;
        const double ar1 = disk_area(b.l1), ar2 = disk_area(b.l2), ar3 = disk_area(b.l3);
        if (INNER) {
            ok = ok && clear_same(b.h1, b.h3, sides_inner(b.ll, b.h1, b.h3)) &&
                 clear_same(b.l1, b.l3, sides_inner(b.lh, b.l1, b.l3)) && clear_mixed_hi(b.ll, b.lh, b.h2, b.h3) &&
                 clear_mixed_lo(b.ll, b.l2, b.l1) && clear_mixed_lo(b.ll, b.l2, b.l3);
            c12_hi = mixed_hi(b.ll, b.lh, b.h2, b.h1, ok);
            c13_hi = inner_angle(b.ll, b.h1, b.h3);
        } else {
            ok = ok && clear_same(b.h1, b.h3, sides_outer(b.h1, b.h3)) &&
                 clear_same(b.l1, b.l3, sides_outer(b.l1, b.l3)) && clear_mixed_hi(b.ll, b.lh, b.h3, b.h2) &&
                 clear_mixed_lo(b.ll, b.l1, b.l2) && clear_mixed_lo(b.ll, b.l3, b.l2);
            c12_hi = mixed_hi(b.ll, b.lh, b.h1, b.h2, ok);
            c13_hi = outer_angle(b.h1, b.h3);
        }
        fa = less_(0.5 * (ar1 + ar2), k * c12_hi, t.tol, ok);
        fb = less_(fma_(0.5, ar1 + ar3, ar2), k * c13_hi, t.tol, ok);
    }
    if (!ok) return 0;
    if (!fa && !fb) return 0;
    if (NEED < NEED_MASK && fa && fb) return 3;
    const FBox b = ref.load();
    uint8_t m = 0;
    if (fa) {
        // g1: c13.lo <= (c12 + c23).hi, often by c13.lo <= c13.hi < c12.hi alone
        bool g1 = c13_hi + kTau < c12_hi;
        if (!g1) {
            const double c13_lo = INNER ? inner_angle(b.lh, b.l1, b.l3) : outer_angle(b.l1, b.l3);
            g1 = c13_lo + kTau < c12_hi;
            if (!g1) {
                const double c23_hi =
                    INNER ? mixed_hi(b.ll, b.lh, b.h2, b.h3, ok) : mixed_hi(b.ll, b.lh, b.h3, b.h2, ok);
                g1 = less_(c13_lo, c12_hi + c23_hi, kTau, ok);
            }
        }
        if (g1) m |= 1;
        if (NEED != NEED_FULL && m) return m;
    }
    if (fb) {
        const double c12_lo = INNER ? mixed_lo(b.ll, b.lh, b.l2, b.l1, ok) : mixed_lo(b.ll, b.lh, b.l1, b.l2, ok);
        const double c23_lo = INNER ? mixed_lo(b.ll, b.lh, b.l2, b.l3, ok) : mixed_lo(b.ll, b.lh, b.l3, b.l2, ok);
        if (!less_(c13_hi, c12_lo + c23_lo, kTau, ok)) m |= 2;
    }
    return m;
}

// end_configuration.cu:71-101
template <bool INNER, class Ref>
CPF_HD bool end2d_fails(const Ref& ref, bool& ok) {
    double lhs, rho, used, other, tol;
    {
        const FBox b = ref.load();
        const Terms t(b);
        tol = t.tol;
        ok = ok && (INNER ? clear_mixed_lo(b.ll, b.l2, b.l1) : clear_mixed_lo(b.ll, b.l1, b.l2));
        const double ca_hi =
            INNER ? mixed_hi(b.ll, b.lh, b.h2, b.h1, ok) : mixed_hi(b.ll, b.lh, b.h1, b.h2, ok);
        const double sa_hi = INNER ? semi_outer(b.h2) : semi_inner(b.ll, b.h2);
        other = INNER ? semi_inner(b.ll, b.h1) : semi_outer(b.h1);
        const double q = INNER ? 1.0 - 2.0 * b.h2 : fma_(2.0, b.h2, b.lh);
        rho = INNER ? q * q - b.lh * b.lh : 1.0 - q * q;
        if (rho < 0.0) rho = 0.0;
        const double a_hi = ca_hi + sa_hi;
        used = 0.5 * t.ratio * a_hi;
        lhs = fma_(0.5, disk_area(b.l1), disk_area(b.l2));
        // reusable = 0.5 rho (a.lo - other), a.lo in [0, a.hi]
        if (!ok) return false;
        if (lhs - kRatio * fma_(0.5 * rho, other, used) > tol) return false;
        if (lhs - kRatio * fma_(0.5 * rho, other - a_hi, used) < -tol) return true;
    }
    const FBox b = ref.load();
    const double a_lo = INNER ? mixed_lo(b.ll, b.lh, b.l2, b.l1, ok) + semi_outer(b.l2)
                              : mixed_lo(b.ll, b.lh, b.l1, b.l2, ok) + semi_inner(b.lh, b.l2);
    return less_(lhs, kRatio * fma_(0.5 * rho, other - a_lo, used), tol, ok);
}

// end_configuration.cu:154-210.  The area test comes first: a handle whose test holds
// does not fail, whatever its early exit (a12 + a23 definitely at least a13) says.
// alpha = (a13 + a3).lo - (a12 + a2).hi is at most (a13 + a3).hi - a2.hi, which often
// shows the failure without a12.
template <bool INNER, class Ref>
CPF_HD bool end3d_fails(const Ref& ref, bool& ok) {
    double a13_hi;
    {
        const FBox b = ref.load();
        const Terms t(b);
        if (INNER) {
            ok = ok && clear_same(b.h1, b.h3, sides_inner(b.ll, b.h1, b.h3)) &&
                 clear_same_low(b.l1, b.l3, sides_inner(b.lh, b.l1, b.l3)) && clear_mixed_hi(b.ll, b.lh, b.h2, b.h1) &&
                 clear_mixed_hi(b.ll, b.lh, b.h2, b.h3) && clear_mixed_lo(b.ll, b.l2, b.l1) &&
                 clear_mixed_lo(b.ll, b.l2, b.l3);
            if (!ok) return false;
            a13_hi = inner_angle(b.ll, b.h1, b.h3);
        } else {
            ok = ok && clear_same(b.h1, b.h3, sides_outer(b.h1, b.h3)) &&
                 clear_same_low(b.l1, b.l3, sides_outer(b.l1, b.l3)) && clear_mixed_hi(b.ll, b.lh, b.h1, b.h2) &&
                 clear_mixed_hi(b.ll, b.lh, b.h3, b.h2) && clear_mixed_lo(b.ll, b.l1, b.l2) &&
                 clear_mixed_lo(b.ll, b.l3, b.l2);
            if (!ok) return false;
            a13_hi = outer_angle(b.h1, b.h3);
        }
        const double a3_hi = INNER ? semi_inner(b.ll, b.h3) : semi_outer(b.h3);
        const double a2_hi = INNER ? semi_outer(b.h2) : semi_inner(b.ll, b.h2);
        const double q = INNER ? fma_(2.0, b.h3, b.lh) : 1.0 - 2.0 * b.h3;
        double rho = INNER ? 1.0 - q * q : q * q - b.lh * b.lh;
        if (rho < 0.0) rho = 0.0;
        const double top = a13_hi + a3_hi, used = 0.5 * t.ratio * top;
        const double lhs = fma_(0.5, disk_area(b.l1), disk_area(b.l2) + disk_area(b.l3));
        if (lhs - kRatio * fma_(-0.5 * rho, top - a2_hi, used) >= -t.tol) {
            const double a13_lo = INNER ? inner_angle(b.lh, b.l1, b.l3) : outer_angle(b.l1, b.l3);
            const double a12_hi = INNER ? mixed_hi(b.ll, b.lh, b.h2, b.h1, ok) : mixed_hi(b.ll, b.lh, b.h1, b.h2, ok);
            const double a3_lo = INNER ? semi_inner(b.lh, b.l3) : semi_outer(b.l3);
            const double alpha = (a13_lo + a3_lo) - (a12_hi + a2_hi);
            const double tol = b.l3 < kMinB ? fma_(0.5 * kLowSlack, rho, t.tol) : t.tol;
            if (!less_(lhs, kRatio * fma_(-0.5 * rho, alpha, used), tol, ok) || !ok) return false;
        }
    }
    const FBox b = ref.load();
    const double s_lo = INNER ? mixed_lo(b.ll, b.lh, b.l2, b.l1, ok) + mixed_lo(b.ll, b.lh, b.l2, b.l3, ok)
                              : mixed_lo(b.ll, b.lh, b.l1, b.l2, ok) + mixed_lo(b.ll, b.lh, b.l3, b.l2, ok);
    return !less_(a13_hi, s_lo, kTau, ok);
}

// start_configuration.cu:126-162.  Criterion 1 is evaluated when a12 + a23 > a13
// possibly holds, criterion 2 unless it definitely holds; "definitely" implies
// "possibly".
template <int NEED, class Ref>
CPF_HD bool start_box(const Ref& ref, FOut& o) {
    bool ok, f1, f2;
    double a12_hi, a13_hi;
    {
        const FBox b = ref.load();
        ok = clear_same(b.h1, b.h3, sides_outer(b.h1, b.h3)) && clear_same(b.l1, b.l3, sides_outer(b.l1, b.l3)) &&
             clear_mixed_hi(b.ll, b.lh, b.h3, b.h2) && clear_mixed_lo(b.ll, b.l1, b.l2) &&
             clear_mixed_lo(b.ll, b.l3, b.l2);
        if (!ok) return false;
        const Terms t(b);
        const double so = semi_outer(b.h1), k = 0.5 * kRatio * t.ratio;
        a12_hi = mixed_hi(b.ll, b.lh, b.h1, b.h2, ok);
        a13_hi = outer_angle(b.h1, b.h3);
        const double ar1 = disk_area(b.l1), ar2 = disk_area(b.l2), ar3 = disk_area(b.l3);
        f1 = less_(fma_(0.5, ar2, ar1), k * (so + a12_hi), t.tol, ok);
        f2 = less_(fma_(0.5, ar3, ar1 + ar2), k * (so + a13_hi), t.tol, ok);
    }
    if (!ok) return false;
    if (NEED < NEED_MASK && f1 && f2) {
        o.mask = 1;
        return true;
    }
    if (NEED != NEED_HANDLES && !f1 && !f2) return true;
    // a13.lo <= a13.hi < a12.hi <= (a12 + a23).hi: "possibly" without a13.lo and a23
    bool pos = a13_hi + kTau < a12_hi, def = false;
    if (pos && f1 && !f2) {
        o.mask = 1;
        return true;
    }
    const FBox b = ref.load();
    if (f2 || (NEED == NEED_HANDLES && !f1)) {
        def = less_(a13_hi, mixed_lo(b.ll, b.lh, b.l1, b.l2, ok) + mixed_lo(b.ll, b.lh, b.l3, b.l2, ok), kTau, ok);
        if (!ok) return false;
        if (def) pos = true;
    }
    if ((f1 || NEED == NEED_HANDLES) && !pos) {
        const double a13_lo = outer_angle(b.l1, b.l3);
        pos = a13_lo + kTau < a12_hi;
        if (!pos) pos = less_(a13_lo, a12_hi + mixed_hi(b.ll, b.lh, b.h3, b.h2, ok), kTau, ok);
    }
    if (pos && f1) o.mask |= 1;
    if (NEED != NEED_FULL && o.mask) return ok;
    if (!def && f2) o.mask |= 2;
    // (where only criterion 1 fails, one is evaluated: it, or criterion 2)
    if (!f1) o.handles = (pos ? 1 : 0) + (def ? 0 : 1);
    return ok;
}

// start_configuration.cu:169-188.  The reused angle lies between 0 and a12.hi + a2.hi - a1.
template <class Ref>
CPF_HD bool start_end_2d_box(const Ref& ref, FOut& o) {
    bool ok;
    double a1, rho, used, lhs, tol;
    {
        const FBox b = ref.load();
        const Terms t(b);
        tol = t.tol;
        // (the order of the mixed corner, before any angle: slabs near lambda = 0.99 that are
        // wide against their disks fail it throughout)
        ok = clear_mixed_lo(b.ll, b.l1, b.l2) && b.lh + b.h2 <= 1.0 - b.h1;
        if (!ok) return false;
        a1 = semi_outer(b.h1);
        const double a2_hi = semi_inner(b.ll, b.h2), a12_hi = mixed_hi(b.ll, b.lh, b.h1, b.h2, ok);
        const double q = fma_(2.0, b.h2, b.lh);
        rho = 1.0 - q * q;
        if (rho < 0.0) rho = 0.0;
        used = 0.5 * t.ratio * (a1 + a2_hi + a12_hi);
        lhs = disk_area(b.l1) + disk_area(b.l2);
        if (!ok) return false;
        if (lhs - kRatio * used > tol) return true;
        double top = a12_hi + a2_hi - a1;
        if (top < 0.0) top = 0.0;
        if (lhs - kRatio * fma_(-0.5 * rho, top, used) < -tol) {
            o.mask = 1;
            return true;
        }
    }
    const FBox b = ref.load();
    double reuse = mixed_lo(b.ll, b.lh, b.l1, b.l2, ok) + semi_inner(b.lh, b.l2) - a1;
    if (reuse < 0.0) reuse = 0.0;
    if (less_(lhs, kRatio * fma_(-0.5 * rho, reuse, used), tol, ok)) o.mask = 1;
    return ok;
}

// start_configuration.cu:227-265 (a13 of r1 and r2, as there).  The reused angle
// a.lo - a122.hi lies between 0 and a.hi - a122.hi.
template <class Ref>
CPF_HD bool start_end_3d_box(const Ref& ref, FOut& o) {
    bool ok;
    double a122_hi, lane, used, lhs, tol;
    {
        const FBox b = ref.load();
        ok = clear_same(b.h1, b.h2, sides_outer(b.h1, b.h2)) && clear_same(b.l1, b.l2, sides_outer(b.l1, b.l2)) &&
             clear_mixed_lo(b.ll, b.l1, b.l2) && clear_mixed_lo(b.ll, b.l3, b.l2);
        if (!ok) return false;
        const Terms t(b);
        tol = t.tol;
        const double a1_hi = semi_outer(b.h1), a2_hi = semi_inner(b.ll, b.h2), a3_hi = semi_outer(b.h3);
        const double a12_hi = mixed_hi(b.ll, b.lh, b.h1, b.h2, ok), a13_hi = outer_angle(b.h1, b.h2);
        const double a23_hi = mixed_hi(b.ll, b.lh, b.h3, b.h2, ok);
        const double b123_hi = a12_hi + a23_hi, b13_hi = a13_hi < b123_hi ? b123_hi : a13_hi;
        const double a123_hi = a1_hi + b13_hi + a3_hi;
        a122_hi = a1_hi + a12_hi + a2_hi;
        const double a_hi = a123_hi < a122_hi ? a122_hi : a123_hi;
        const double outer = fma_(-2.0, b.h3, 1.0);
        lane = 0.5 * (outer * outer - b.lh * b.lh);
        if (lane < 0.0) lane = 0.0;
        used = 0.5 * t.ratio * a_hi;
        lhs = disk_area(b.l1) + (disk_area(b.l2) + disk_area(b.l3));
        if (!ok) return false;
        if (lhs - kRatio * used > tol) return true;
        if (lhs - kRatio * fma_(-lane, a_hi - a122_hi, used) < -tol) {
            o.mask = 1;
            return true;
        }
    }
    const FBox b = ref.load();
    const double a1_lo = semi_outer(b.l1), a2_lo = semi_inner(b.lh, b.l2), a3_lo = semi_outer(b.l3);
    const double a12_lo = mixed_lo(b.ll, b.lh, b.l1, b.l2, ok), a13_lo = outer_angle(b.l1, b.l2);
    const double b123_lo = a12_lo + mixed_lo(b.ll, b.lh, b.l3, b.l2, ok);
    const double b13_lo = a13_lo < b123_lo ? b123_lo : a13_lo;
    const double a123_lo = a1_lo + b13_lo + a3_lo, a122_lo = a1_lo + a12_lo + a2_lo;
    double reuse = (a123_lo < a122_lo ? a122_lo : a123_lo) - a122_hi;
    if (reuse < 0.0) reuse = 0.0;
    if (less_(lhs, kRatio * fma_(-lane, reuse, used), tol, ok)) o.mask = 1;
    return ok;
}

// The verdict of a box that is neither empty nor stopped by the fit check.  order:
// bit 0 = second handle first (DECIDE).  Returns false when the box is left to
// eval_box; else o holds what NEED asks for.
template <int FAM, int NEED, class Ref>
CPF_HD bool filter_box(const Ref& ref, int order, FOut& o) {
    constexpr bool kThree = FAM != 1 && FAM != 4;
    if (!box_ok<kThree>(ref.load())) return false;
    o.mask = 0;
    o.handles = 1;
    if (FAM == 0) return start_box<NEED>(ref, o);
    if (FAM == 1) return start_end_2d_box(ref, o);
    if (FAM == 2) return start_end_3d_box(ref, o);
    const bool second = NEED != NEED_FULL && (order & 1);
    bool ok = true;
    uint8_t h = 0;
    for (int i = 0; i < 2; ++i) {
        const bool inner = (i == 0) != second;
        ++h;
        uint8_t m;
        if (FAM == 3)
            m = inner ? middle_handle<NEED, true>(ref, ok) : (uint8_t)(middle_handle<NEED, false>(ref, ok) << 2);
        else if (FAM == 4)
            m = inner ? (end2d_fails<true>(ref, ok) ? 1 : 0) : (end2d_fails<false>(ref, ok) ? 2 : 0);
        else
            m = inner ? (end3d_fails<true>(ref, ok) ? 1 : 0) : (end3d_fails<false>(ref, ok) ? 2 : 0);
        if (!ok) return false;
        o.mask |= m;
        if (NEED != NEED_FULL && m) break;
    }
    o.handles = h;
    return true;
}

}  // namespace flt
}  // namespace cpb
