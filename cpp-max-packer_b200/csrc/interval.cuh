// Outward-rounded FP64 interval arithmetic shared by host and device.
//
// Restates the raster interval primitives of the reference
// (engine/pack_geometry/src/validation_kernel.cpp:291-324 widened/add/
// subtract/multiply/divide, :1942-1966 interval vector ops, :2038-2079
// triangle_box_disjoint, :2081-2100 grid_cell_interval) so that device and
// host results are bit-identical to it: every operation is one IEEE binary64
// round-to-nearest operation (device: __dadd_rn/__dmul_rn/... so nothing is
// contracted into an FMA), then each bound moves one ulp outward with an
// integer-bit nextafter; min/max keep std::min/std::max semantics.
#pragma once

#include <cstdint>
#include <cstring>

#include "common.cuh"

namespace spk {

SPK_HD double f_add(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
SPK_HD double f_sub(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __dsub_rn(a, b);
#else
    return a - b;
#endif
}
SPK_HD double f_mul(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
SPK_HD double f_div(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __ddiv_rn(a, b);
#else
    return a / b;
#endif
}

SPK_HD std::uint64_t f_bits(double v)
{
#ifdef __CUDA_ARCH__
    return static_cast<std::uint64_t>(__double_as_longlong(v));
#else
    std::uint64_t b;
    std::memcpy(&b, &v, 8);
    return b;
#endif
}
SPK_HD double f_from_bits(std::uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double(static_cast<long long>(b));
#else
    double v;
    std::memcpy(&v, &b, 8);
    return v;
#endif
}

SPK_HD bool f_finite(double v) { return (f_bits(v) & 0x7ff0000000000000ULL) != 0x7ff0000000000000ULL; }

// IEEE nextafter(v, +inf) from the bit representation (the next representable
// binary64 value in that direction).
SPK_HD double next_up(double v)
{
    if (v != v) {
        return v;
    }
    const std::uint64_t b = f_bits(v);
    if ((b & 0x7fffffffffffffffULL) == 0) {
        return f_from_bits(0x0000000000000001ULL);  // +denorm_min
    }
    if (b >> 63) {
        return f_from_bits(b - 1);
    }
    return b == 0x7ff0000000000000ULL ? v : f_from_bits(b + 1);
}

// std::min / std::max semantics: min(a, b) = (b < a) ? b : a.
SPK_HD double f_min(double a, double b) { return (b < a) ? b : a; }
SPK_HD double f_max(double a, double b) { return (a < b) ? b : a; }

struct Interval {
    double low;
    double high;
    bool valid;
};

SPK_HD Interval point_interval(double v) { return { v, v, f_finite(v) }; }

// The representable values next below and above a finite v.  Like the interval operations below
// without branches: neighbouring threads' signs differ, and a branch per bound
// cost the device more than the operations themselves.
SPK_HD double finite_down(double v)
{
    const std::uint64_t b = f_bits(v), negative = b >> 63;
    const std::uint64_t r = b - 1 + 2 * negative;
    return f_from_bits((b << 1) == 0 ? 0x8000000000000001ULL : r);
}
SPK_HD double finite_up(double v)
{
    const std::uint64_t b = f_bits(v), negative = b >> 63;
    const std::uint64_t r = b + 1 - 2 * negative;
    return f_from_bits((b << 1) == 0 ? 0x0000000000000001ULL : r);
}

SPK_HD Interval interval_if(bool keep, Interval v) { return { keep ? v.low : 0.0, keep ? v.high : 0.0, keep && v.valid }; }

SPK_HD Interval widened(double low, double high)
{
    const double l = finite_down(low), h = finite_up(high);
    const bool valid = f_finite(l) & f_finite(h);
    return interval_if(f_finite(low) & f_finite(high), { l, h, valid });
}

SPK_HD Interval add_interval(Interval a, Interval b)
{
    return interval_if(a.valid & b.valid, widened(f_add(a.low, b.low), f_add(a.high, b.high)));
}

SPK_HD Interval subtract_interval(Interval a, Interval b)
{
    return interval_if(a.valid & b.valid, widened(f_sub(a.low, b.high), f_sub(a.high, b.low)));
}

SPK_HD Interval multiply_interval(Interval a, Interval b)
{
    const double v0 = f_mul(a.low, b.low), v1 = f_mul(a.low, b.high), v2 = f_mul(a.high, b.low),
                 v3 = f_mul(a.high, b.high);
    const bool keep = a.valid & b.valid & f_finite(v0) & f_finite(v1) & f_finite(v2) & f_finite(v3);
    // std::ranges::min_element / max_element: the first minimum / maximum.
    const double lo = f_min(f_min(f_min(v0, v1), v2), v3), hi = f_max(f_max(f_max(v0, v1), v2), v3);
    return interval_if(keep, widened(lo, hi));
}

// multiply_interval(a, point_interval(p)).  With a point operand the four
// products are two, each computed twice, and the first-minimum / first-maximum
// scan picks the same values from the pair, so the result is identical.
SPK_HD Interval multiply_by_point(const Interval& a, double p)
{
    const double v0 = f_mul(a.low, p), v2 = f_mul(a.high, p);
    const bool keep = a.valid & f_finite(p) & f_finite(v0) & f_finite(v2);
    return interval_if(keep, widened(f_min(v0, v2), f_max(v0, v2)));
}

// transformed_interval (validation_kernel.cpp:805-943): row `row` of the
// rotation intervals applied to a point, plus the translation, as intervals.
// Host and device run this same code.
SPK_HD Interval transformed_interval_at(const double* point, const double* translation, const Interval (*rotation)[3],
                                        int row)
{
    Interval value = point_interval(translation[row]);
    for (int column = 0; column < 3; ++column) {
        value = add_interval(value, multiply_by_point(rotation[row][column], point[column]));
    }
    return value;
}

SPK_HD Interval divide_interval(Interval n, Interval d)
{
    if (!n.valid || !d.valid || d.low <= 0.0) {
        return { 0, 0, false };
    }
    const Interval reciprocal = widened(f_div(1.0, d.high), f_div(1.0, d.low));
    return multiply_interval(n, reciprocal);
}

struct IVec3 {
    Interval v[3];
};

SPK_HD IVec3 ivec_sub(const IVec3& a, const IVec3& b)
{
    return { { subtract_interval(a.v[0], b.v[0]), subtract_interval(a.v[1], b.v[1]),
               subtract_interval(a.v[2], b.v[2]) } };
}

SPK_HD IVec3 ivec_cross(const IVec3& a, const IVec3& b)
{
    return { { subtract_interval(multiply_interval(a.v[1], b.v[2]), multiply_interval(a.v[2], b.v[1])),
               subtract_interval(multiply_interval(a.v[2], b.v[0]), multiply_interval(a.v[0], b.v[2])),
               subtract_interval(multiply_interval(a.v[0], b.v[1]), multiply_interval(a.v[1], b.v[0])) } };
}

SPK_HD Interval ivec_dot(const IVec3& a, const IVec3& b)
{
    Interval r = point_interval(0.0);
    for (int i = 0; i < 3; ++i) {
        r = add_interval(r, multiply_interval(a.v[i], b.v[i]));
    }
    return r;
}

SPK_HD bool projection_separates(const IVec3* tri, const IVec3& box, const IVec3& axis)
{
    Interval tp = ivec_dot(tri[0], axis);
#pragma unroll
    for (int k = 1; k < 3; ++k) {
        const Interval p = ivec_dot(tri[k], axis);
        if (!p.valid) {
            return false;
        }
        tp.low = f_min(tp.low, p.low);
        tp.high = f_max(tp.high, p.high);
    }
    const Interval bp = ivec_dot(box, axis);
    return tp.valid && bp.valid && (tp.high < bp.low || bp.high < tp.low);
}

// 13-axis separating-axis test of a triangle (vertex intervals) and a box.
SPK_HD bool triangle_box_disjoint(const IVec3* tri, const IVec3& box)
{
    // The axis loops are unrolled so that their array indices are constants
    // and the intervals stay in registers; the operations and their order are
    // as written.
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double lo = tri[0].v[a].low, hi = tri[0].v[a].high;
#pragma unroll
        for (int k = 1; k < 3; ++k) {
            lo = f_min(lo, tri[k].v[a].low);
            hi = f_max(hi, tri[k].v[a].high);
        }
        if (hi < box.v[a].low || box.v[a].high < lo) {
            return true;
        }
    }
    const IVec3 first = ivec_sub(tri[1], tri[0]);
    const IVec3 second = ivec_sub(tri[2], tri[0]);
    if (projection_separates(tri, box, ivec_cross(first, second))) {
        return true;
    }
    const IVec3 edges[3] = { first, second, ivec_sub(tri[2], tri[1]) };
    // The edge loop stays rolled: nine unrolled axis tests made the raster
    // wait on instruction fetch (measured faster rolled, at six blocks per SM).
#pragma unroll 1
    for (int e = 0; e < 3; ++e) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            IVec3 axis = { { point_interval(0.0), point_interval(0.0), point_interval(0.0) } };
            axis.v[a] = point_interval(1.0);
            if (projection_separates(tri, box, ivec_cross(edges[e], axis))) {
                return true;
            }
        }
    }
    return false;
}

// The parts of triangle_box_disjoint that depend on the triangle alone, for
// rasterising one triangle against many cells: the triangle's bounds on the
// three box axes, the ten remaining axes (normal, then edge e x unit axis a
// for e, a = 0..2, the test order) and the triangle's projection on each.
// face_sat_disjoint(f, box) with f from face_sat(tri, f) returns exactly
// triangle_box_disjoint(tri, box): every value is the same expression
// computed once instead of once per cell.
struct FaceSat {
    double lo[3], hi[3];
    IVec3 axis[10];
    double tp_low[10], tp_high[10];
    unsigned char usable[10];  // axis i can separate (all three vertex projections valid)
};

// FaceSat's box-axis bounds.
SPK_HD void face_sat_bounds(const IVec3* tri, FaceSat& f)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double lo = tri[0].v[a].low, hi = tri[0].v[a].high;
#pragma unroll
        for (int k = 1; k < 3; ++k) {
            lo = f_min(lo, tri[k].v[a].low);
            hi = f_max(hi, tri[k].v[a].high);
        }
        f.lo[a] = lo;
        f.hi[a] = hi;
    }
}

// FaceSat's axis i (0: the normal first x second; 1 + 3 e + a: edge e x
// unit axis a, with edges first = v1 - v0, second = v2 - v0, v2 - v1) and the
// triangle's projection on it.  Each axis is independent of the others, so a
// device launch gives each its own thread.
SPK_HD void face_sat_axis(const IVec3* tri, int i, FaceSat& f)
{
    // The normal is the cross product of the first two edges, the others of an
    // edge and a unit vector: one expression, so that threads do not diverge.
    const IVec3 e0 = ivec_sub(tri[1], tri[0]), e1 = ivec_sub(tri[2], tri[0]), e2 = ivec_sub(tri[2], tri[1]);
    const int e = (i + 2) / 3 - 1, a = (i + 2) % 3;  // of axes 1 to 9
    IVec3 second = { { point_interval(0.0), point_interval(0.0), point_interval(0.0) } };
    second.v[a] = point_interval(1.0);
    const IVec3 axis = ivec_cross(i < 4 ? e0 : e == 1 ? e1 : e2, i == 0 ? e1 : second);
    f.axis[i] = axis;
    // projection_separates' triangle side: false whenever a vertex
    // projection is invalid, whatever the box.
    Interval tp = ivec_dot(tri[0], axis);
    bool usable = tp.valid;
    for (int k = 1; k < 3 && usable; ++k) {
        const Interval p = ivec_dot(tri[k], axis);
        if (!p.valid) {
            usable = false;
            break;
        }
        tp.low = f_min(tp.low, p.low);
        tp.high = f_max(tp.high, p.high);
    }
    f.tp_low[i] = tp.low;
    f.tp_high[i] = tp.high;
    f.usable[i] = usable ? 1 : 0;
}

SPK_HD void face_sat(const IVec3* tri, FaceSat& f)
{
    face_sat_bounds(tri, f);
    for (int i = 0; i < 10; ++i) {
        face_sat_axis(tri, i, f);
    }
}

SPK_HD bool face_sat_disjoint(const FaceSat& f, const IVec3& box)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (f.hi[a] < box.v[a].low || box.v[a].high < f.lo[a]) {
            return true;
        }
    }
#pragma unroll 1
    for (int i = 0; i < 10; ++i) {
        if (!f.usable[i]) {
            continue;
        }
        const Interval bp = ivec_dot(box, f.axis[i]);
        if (bp.valid && (f.tp_high[i] < bp.low || bp.high < f.tp_low[i])) {
            return true;
        }
    }
    return false;
}

// A filter in plain binary64 before the interval test: the separating-axis test
// of the vertex intervals' midpoints and the cell's centre and half edge, with
// margins far above what interval widths and rounding can move a projection.
// Where an axis' gap lies beyond its margin the interval test separates there;
// where no axis' gap comes within its margin of separating, it separates
// nowhere; the rest goes to the interval test.
//
// With u = 2^-53, C a bound on every coordinate, W on the widths of the vertex
// intervals, e on the edges' components and D = W + 32 u C: the interval
// test's projections on an edge axis stray from the real ones by less than 24 C
// W + 96 u C e and the filter's by less than 30 C D, 60 C D in all (e <= 2 C);
// on the normal by less than 144 C e D; the box axes by less than 4 D.  The
// margins are 256 C D, 1024 C e D and 256 D.
struct FaceFilter {
    double v[3][3];     // vertex midpoints
    double e[3][3];     // v1 - v0, v2 - v0, v2 - v1
    double n[3];        // e0 x e1
    double box_margin, edge_margin, normal_margin;
    bool usable;
};

// `reach`: a bound on the lattice's |origin| and on the distance from the
// triangle's bounds to any cell that will be tested.
SPK_HD void face_filter(const IVec3* tri, double reach, FaceFilter& f)
{
    double most = 0.0, width = 0.0;
    f.usable = true;
    for (int k = 0; k < 3; ++k) {
        for (int a = 0; a < 3; ++a) {
            const Interval& i = tri[k].v[a];
            f.usable = f.usable && i.valid;
            f.v[k][a] = 0.5 * (i.low + i.high);
            const double m = f_max(i.low < 0 ? -i.low : i.low, i.high < 0 ? -i.high : i.high);
            most = f_max(most, m);
            width = f_max(width, i.high - i.low);
        }
    }
    const double C = 2.0 * (most + reach);
    const double D = width + 0x1p-48 * C;
    double edge = 0.0;
    for (int a = 0; a < 3; ++a) {
        f.e[0][a] = f.v[1][a] - f.v[0][a];
        f.e[1][a] = f.v[2][a] - f.v[0][a];
        f.e[2][a] = f.v[2][a] - f.v[1][a];
        for (int k = 0; k < 3; ++k) {
            edge = f_max(edge, f.e[k][a] < 0 ? -f.e[k][a] : f.e[k][a]);
        }
    }
    f.n[0] = f.e[0][1] * f.e[1][2] - f.e[0][2] * f.e[1][1];
    f.n[1] = f.e[0][2] * f.e[1][0] - f.e[0][0] * f.e[1][2];
    f.n[2] = f.e[0][0] * f.e[1][1] - f.e[0][1] * f.e[1][0];
    f.box_margin = 256.0 * D + 1e-290;
    f.edge_margin = 256.0 * C * D + 1e-290;
    f.normal_margin = 1024.0 * C * (edge + D) * D + 1e-290;
    // Magnitudes whose products stay far from the ends of the range.
    f.usable = f.usable && C < 1e75 && C > 1e-75;
}

SPK_HD double gap_of(double p, double q, double r)
{
    const double lo = p < q ? p : q, hi = p < q ? q : p;
    return (lo > -hi ? lo : -hi) - r;
}

enum class FaceCell { disjoint, meets, uncertain };

// The cell with centre c and half edge h.
SPK_HD FaceCell face_filter_cell(const FaceFilter& f, const double* c, double h)
{
    if (!f.usable) {
        return FaceCell::uncertain;
    }
    double w[3][3];
    bool near = false;
    for (int a = 0; a < 3; ++a) {
        for (int k = 0; k < 3; ++k) {
            w[k][a] = f.v[k][a] - c[a];
        }
        const double lo = f_min(f_min(w[0][a], w[1][a]), w[2][a]), hi = f_max(f_max(w[0][a], w[1][a]), w[2][a]);
        const double g = gap_of(lo, hi, h);
        if (g > f.box_margin) {
            return FaceCell::disjoint;
        }
        near = near || g >= -f.box_margin;
    }
    {
        const double d = f.n[0] * w[0][0] + f.n[1] * w[0][1] + f.n[2] * w[0][2];
        const double r = h * ((f.n[0] < 0 ? -f.n[0] : f.n[0]) + (f.n[1] < 0 ? -f.n[1] : f.n[1]) +
                              (f.n[2] < 0 ? -f.n[2] : f.n[2]));
        const double g = gap_of(d, d, r);
        if (g > f.normal_margin) {
            return FaceCell::disjoint;
        }
        near = near || g >= -f.normal_margin;
    }
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        // Both ends of the edge project alike; `o` is the vertex opposite.
        const int s = e == 2 ? 1 : 0, o = 2 - e;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int b = (a + 1) % 3, d = (a + 2) % 3;  // the axis is (edge_d, -edge_b) over (b, d)
            const double eb = f.e[e][b], ed = f.e[e][d];
            const double p = ed * w[s][b] - eb * w[s][d], q = ed * w[o][b] - eb * w[o][d];
            const double r = h * ((eb < 0 ? -eb : eb) + (ed < 0 ? -ed : ed));
            const double g = gap_of(p, q, r);
            if (g > f.edge_margin) {
                return FaceCell::disjoint;
            }
            near = near || g >= -f.edge_margin;
        }
    }
    return near ? FaceCell::uncertain : FaceCell::meets;
}

// Outward enclosure of the closed cell `index` on the lattice; false when an
// index is not exactly representable (|index| >= 2^53) or arithmetic overflows.
SPK_HD bool grid_cell_interval(const double* origin, double pitch, const std::int64_t* index, IVec3& out)
{
    const std::int64_t limit = std::int64_t { 1 } << 53;
    for (int a = 0; a < 3; ++a) {
        if (index[a] < -limit || index[a] >= limit) {
            return false;
        }
        const Interval low = add_interval(point_interval(origin[a]),
                                          multiply_interval(point_interval(pitch),
                                                            point_interval(static_cast<double>(index[a]))));
        const Interval high = add_interval(point_interval(origin[a]),
                                           multiply_interval(point_interval(pitch),
                                                             point_interval(static_cast<double>(index[a] + 1))));
        if (!low.valid || !high.valid) {
            return false;
        }
        out.v[a] = { f_min(low.low, high.low), f_max(low.high, high.high), true };
    }
    return true;
}

}  // namespace spk
