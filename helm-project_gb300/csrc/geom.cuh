// FP64 spherical geometry on the device. Every expression keeps the
// operation order of the reference (libs/axis/include/axis/detail/
// spherical_clipper.hpp:39-335) and the translation units that include
// this header are compiled with --fmad=false, so additions and products
// round exactly as the reference's host build does; sqrt and division are
// IEEE round-to-nearest on the device as on the host. Only atan2/acos come
// from CUDA's libdevice and may differ from the host libm by an ulp.
#pragma once

#include <cstdint>

namespace axgb {

struct DV3 {
    double x, y, z;
};

__device__ __forceinline__ double d_dot(const DV3 &a, const DV3 &b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ DV3 d_cross(const DV3 &a, const DV3 &b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double d_lensq(const DV3 &v) { return v.x * v.x + v.y * v.y + v.z * v.z; }
__device__ __forceinline__ DV3 d_normalize(const DV3 &v) {
    double len = sqrt(d_lensq(v));
    if (len < 1.0e-300) return {0.0, 0.0, 0.0};
    double inv = 1.0 / len;
    return {v.x * inv, v.y * inv, v.z * inv};
}
__device__ __forceinline__ DV3 d_add(const DV3 &a, const DV3 &b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }

// a / b correctly rounded, from the correctly rounded reciprocal y of b, by
// two corrections with exact FMA residuals (Markstein, IBM J. Res. Dev. 34,
// 1990): five operations where the division takes about 25. Operands outside
// 2^+-500 (and zeros), where the residuals could be inexact, are divided.
__device__ __forceinline__ bool d_mid_range(double v) {
    return static_cast<unsigned>(((__double2hiint(v) >> 20) & 0x7ff) - 523) <= 1000u;
}
__device__ __forceinline__ double d_div_by(double a, double b, double y) {
    if (!d_mid_range(a) || !d_mid_range(b)) return a / b;
    const double q0 = __dmul_rn(a, y);
    const double q1 = __fma_rn(__fma_rn(-b, q0, a), y, q0);
    return __fma_rn(__fma_rn(-b, q1, a), y, q1);
}

// Fixed-capacity polygon in registers/local memory. push() past CAP sets
// `over`; with CAP = 32 this is exactly the reference's silent drop
// (SphericalPolygon::push, spherical_clipper.hpp:145-150), with a smaller
// CAP the caller re-runs the pair at CAP = 32.
template <int CAP>
struct DPoly {
    double x[CAP], y[CAP], z[CAP];
    int n;
    bool over;
    __device__ __forceinline__ void clear() {
        n = 0;
        over = false;
    }
    __device__ __forceinline__ void push(const DV3 &v) {
        if (n < CAP) {
            x[n] = v.x;
            y[n] = v.y;
            z[n] = v.z;
            ++n;
        } else {
            over = true;
        }
    }
    __device__ __forceinline__ DV3 at(int i) const { return {x[i], y[i], z[i]}; }
};

// Van Oosterom-Strackee fan from vertex 0, |sum of 2*atan2|
// (spherical_clipper.hpp:112-137).
template <int CAP>
__device__ double d_poly_area(const DPoly<CAP> &p) {
    if (p.n < 3) return 0.0;
    double total = 0.0;
    DV3 a = p.at(0);
    for (int i = 1; i < p.n - 1; ++i) {
        DV3 b = p.at(i), c = p.at(i + 1);
        double ab = d_dot(a, b);
        double ac = d_dot(a, c);
        double bc = d_dot(b, c);
        DV3 bxc = d_cross(b, c);
        double num = d_dot(a, bxc);
        double den = 1.0 + ab + ac + bc;
        double tri = 2.0 * atan2(num, den);
        total += tri;
    }
    return fabs(total);
}

// Arc (v1 -> v2) against the great circle of normal n1 = ea x eb, midpoint
// fallback (spherical_clipper.hpp:265-295; the caller passes the edge
// normal it already formed, the same product).
__device__ __forceinline__ DV3 d_arc_cross(const DV3 &v1, const DV3 &v2, const DV3 &n1) {
    DV3 n2 = d_cross(v1, v2);
    DV3 d = d_cross(n1, n2);
    double dl = d_lensq(d);
    if (dl < 1.0e-30) return d_normalize(d_add(v1, v2));
    DV3 c = d_normalize(d);
    DV3 mid = d_normalize(d_add(v1, v2));
    if (d_dot(c, mid) < 0.0) c = {-c.x, -c.y, -c.z};
    return c;
}

// The same point, with the two square roots and reciprocals of the midpoint
// test left out where its sign is beyond doubt: |c| = 1 and the midpoint of
// an arc between unit vectors has length at most 2, so the dot products with
// the midpoint and with the normalised midpoint differ from their exact
// values by less than 1e-14, and above 1e-3 they have the same sign.
__device__ __forceinline__ DV3 d_arc_cross_fast(const DV3 &v1, const DV3 &v2, const DV3 &n1) {
    DV3 n2 = d_cross(v1, v2);
    DV3 d = d_cross(n1, n2);
    if (d_lensq(d) < 1.0e-30) return d_normalize(d_add(v1, v2));
    DV3 c = d_normalize(d);
    DV3 mid = d_add(v1, v2);
    double side = d_dot(c, mid);
    if (fabs(side) <= 1.0e-3) side = d_dot(c, d_normalize(mid));
    if (side < 0.0) c = {-c.x, -c.y, -c.z};
    return c;
}

// Ordered as doubles for values that are not negative and not NaN, without
// the FP64 pipe.
__device__ __forceinline__ bool d_less_pos(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }

// The same point where its sign is known beforehand. d = n1 x (v1 x v2) =
// v1 (n1.v2) - v2 (n1.v1): going into the half space (n1.v1 < 0 < n1.v2) both
// factors are positive, so d is on the side of v1 + v2; coming out both are
// negative, and -d is. For arcs under 120 degrees with both ends clear of the
// plane.
__device__ __forceinline__ DV3 d_arc_cross_known(const DV3 &v1, const DV3 &v2, const DV3 &n1, bool out) {
    const DV3 d = d_cross(n1, d_cross(v1, v2));
    const double l2 = d_lensq(d);
    if (d_less_pos(l2, 1.0e-30)) return d_normalize(d_add(v1, v2));
    const double inv = 1.0 / sqrt(l2);
    const DV3 c{d.x * inv, d.y * inv, d.z * inv};
    return out ? DV3{-c.x, -c.y, -c.z} : c;
}

// 2 atan2(num, den) for the small triangles that cells are cut into: up to
// num / den = 2^-7 by Gregory's series to the ninth power (the next term is
// below 2^-73 of the first), so the error is the quotient's rounding and the
// last addition's. The quotient: a float reciprocal, two Newton steps (each
// doubles its 23 bits), one correction with the exact residual. Larger
// angles by atan2.
__device__ __forceinline__ double d_twice_atan(double num, double den) {
    if (static_cast<unsigned>(__double2hiint(den) - 0x3fe00000) < 0x00500000u) {  // 1/2 <= den < 16
        double y = static_cast<double>(__frcp_rn(static_cast<float>(den)));
        y = __fma_rn(__fma_rn(-den, y, 1.0), y, y);
        y = __fma_rn(__fma_rn(-den, y, 1.0), y, y);
        const double q0 = __dmul_rn(num, y);
        const double t = __fma_rn(__fma_rn(-den, q0, num), y, q0), q = t * t;
        if ((__double2hiint(t) & 0x7fffffff) < 0x3f800000) {  // |t| < 2^-7
            const double r = __fma_rn(q, __fma_rn(q, __fma_rn(q, 1.0 / 9.0, -1.0 / 7.0), 1.0 / 5.0), -1.0 / 3.0);
            return 2.0 * __fma_rn(t * q, r, t);
        }
    }
    return 2.0 * atan2(num, den);
}

// Clip `subject` by every edge of `clip` (Sutherland-Hodgman on great
// circles, inclusive eps = -1e-14, edges with |a x b|^2 < 1e-30 skipped;
// spherical_clipper.hpp:181-229 and :301-335). Returns the overlap area;
// sets *over when a polygon exceeded CAP.
// The previous vertex's side test is the value the loop formed one step
// earlier (the same dot product), and the two buffers swap roles per edge.
template <int CAP>
__device__ double d_overlap_area(const DPoly<CAP> &subject, const DPoly<CAP> &clip, DPoly<CAP> &bufa,
                                 DPoly<CAP> &bufb, bool *over) {
    *over = subject.over || clip.over;
    if (subject.n < 3 || clip.n < 3) return 0.0;
    bufa.n = subject.n;
    bufa.over = false;
    for (int i = 0; i < subject.n; ++i) {
        bufa.x[i] = subject.x[i];
        bufa.y[i] = subject.y[i];
        bufa.z[i] = subject.z[i];
    }
    DPoly<CAP> *in = &bufa, *out = &bufb;
    constexpr double eps = -1.0e-14;
    for (int ci = 0; ci < clip.n; ++ci) {
        DV3 ea = clip.at(ci);
        DV3 eb = clip.at(ci + 1 == clip.n ? 0 : ci + 1);
        DV3 nrm = d_cross(ea, eb);
        if (d_lensq(nrm) < 1.0e-30) continue;
        out->clear();
        const int nin = in->n;
        DV3 prv = in->at(nin - 1);
        double dp = d_dot(nrm, prv);
        for (int i = 0; i < nin; ++i) {
            DV3 cur = in->at(i);
            double dc = d_dot(nrm, cur);
            bool cin = dc >= eps;
            bool pin = dp >= eps;
            if (cin) {
                if (!pin) out->push(d_arc_cross(prv, cur, nrm));
                out->push(cur);
            } else if (pin) {
                out->push(d_arc_cross(prv, cur, nrm));
            }
            prv = cur;
            dp = dc;
        }
        if (out->over) *over = true;
        DPoly<CAP> *t = in;
        in = out;
        out = t;
        if (in->n < 3) return 0.0;
    }
    return d_poly_area(*in);
}

// Degenerate classification (degenerate_cell_handler.hpp:115-142, 259-367):
// 0 none, 1 zero area, 2 collapsed, 3 self-intersecting.
template <int CAP>
__device__ int d_classify(const DPoly<CAP> &p, double area) {
    if (p.n < 3) return 1;
    if (area < 1e-25) return 1;
    const double t2 = 1e-15 * 1e-15;
    int uniq = 1;
    for (int i = 1; i < p.n; ++i) {
        bool dup = false;
        for (int j = 0; j < i; ++j) {
            DV3 d{p.x[i] - p.x[j], p.y[i] - p.y[j], p.z[i] - p.z[j]};
            if (d_lensq(d) < t2) {
                dup = true;
                break;
            }
        }
        if (!dup) ++uniq;
    }
    if (uniq < 3) return 2;
    if (p.n >= 4) {
        for (int i = 0; i < p.n; ++i) {
            int in = (i + 1) % p.n;
            for (int j = i + 2; j < p.n; ++j) {
                int jn = (j + 1) % p.n;
                if (jn == i) continue;
                DV3 a = p.at(i), b = p.at(in), c = p.at(j), d = p.at(jn);
                DV3 nab = d_cross(a, b);
                double dc = d_dot(nab, c), dd = d_dot(nab, d);
                if (dc * dd >= 0.0) continue;
                DV3 ncd = d_cross(c, d);
                double da = d_dot(ncd, a), db = d_dot(ncd, b);
                if (da * db >= 0.0) continue;
                return 3;
            }
        }
    }
    return 0;
}

}  // namespace axgb
