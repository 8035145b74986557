/*
 * b2g_shape.cuh — a fixture definition's shape as the kernels read it (ShapeRec), on the host (fixtures
 * of a world) and on the device (the stand-alone time of impact): the same IEEE operations on both, so
 * the same bits.
 */
#ifndef B2G_SHAPE_CUH
#define B2G_SHAPE_CUH

#include "b2g.h"
#include "b2g_internal.h"

namespace b2g {

/* B2polygonShape::set_as_box, private/collision/b2_polygon_shape.rs:12-23 */
B2G_HD void polygon_box(ShapeRec& s, float hx, float hy) {
    s.v[0] = mk(-hx, -hy);
    s.v[1] = mk(hx, -hy);
    s.v[2] = mk(hx, hy);
    s.v[3] = mk(-hx, hy);
    s.n[0] = mk(0.0f, -1.0f);
    s.n[1] = mk(1.0f, 0.0f);
    s.n[2] = mk(0.0f, 1.0f);
    s.n[3] = mk(-1.0f, 0.0f);
    s.centroid = mk(0.0f, 0.0f);
    s.meta = SHAPE_POLYGON | (4 << 8);
}

/* polygon centroid, b2_polygon_shape.rs:53-77 */
B2G_HD V2 polygon_centroid(const V2* vs, int count) {
    V2 c = mk(0.0f, 0.0f);
    float area = 0.0f;
    const V2 s = vs[0];
    const float inv3 = 1.0f / 3.0f;
    for (int i = 0; i < count; ++i) {
        V2 p1 = sub(vs[0], s);
        V2 p2 = sub(vs[i], s);
        V2 p3 = (i + 1 < count) ? sub(vs[i + 1], s) : sub(vs[0], s);
        V2 e1 = sub(p2, p1);
        V2 e2 = sub(p3, p1);
        float d = cross(e1, e2);
        float tri = 0.5f * d;
        area += tri;
        c = add(c, scale(tri * inv3, add(add(p1, p2), p3)));
    }
    return add(scale(fdiv(1.0f, area), c), s);
}

/* B2polygonShape::set (gift wrapping), b2_polygon_shape.rs:96-211; false -> unit box fallback */
B2G_HD bool polygon_hull(ShapeRec& s, const b2g_vec2* in, int count) {
    if (count < 3) {
        polygon_box(s, 1.0f, 1.0f);
        return false;
    }
    int n = count < kMaxPolygonVertices ? count : kMaxPolygonVertices;
    V2 ps[kMaxPolygonVertices];
    int temp = 0;
    for (int i = 0; i < n; ++i) {
        V2 v = mk(in[i].x, in[i].y);
        bool unique = true;
        for (int j = 0; j < temp; ++j) {
            if (dist_sq(v, ps[j]) < ((0.5f * kLinearSlop) * (0.5f * kLinearSlop))) {
                unique = false;
                break;
            }
        }
        if (unique) ps[temp++] = v;
    }
    n = temp;
    if (n < 3) {
        polygon_box(s, 1.0f, 1.0f);
        return false;
    }
    int i0 = 0;
    float x0 = ps[0].x;
    for (int i = 1; i < n; ++i) {
        float x = ps[i].x;
        if (x > x0 || (x == x0 && ps[i].y < ps[i0].y)) {
            i0 = i;
            x0 = x;
        }
    }
    int hull[kMaxPolygonVertices];
    int m = 0, ih = i0;
    for (;;) {
        if (m >= kMaxPolygonVertices) {
            polygon_box(s, 1.0f, 1.0f);
            return false;
        }
        hull[m] = ih;
        int ie = 0;
        for (int j = 1; j < n; ++j) {
            if (ie == ih) {
                ie = j;
                continue;
            }
            V2 r = sub(ps[ie], ps[hull[m]]);
            V2 v = sub(ps[j], ps[hull[m]]);
            float c = cross(r, v);
            if (c < 0.0f) ie = j;
            if (c == 0.0f && length_sq(v) > length_sq(r)) ie = j;
        }
        ++m;
        ih = ie;
        if (ie == i0) break;
    }
    if (m < 3) {
        polygon_box(s, 1.0f, 1.0f);
        return false;
    }
    for (int i = 0; i < m; ++i) s.v[i] = ps[hull[i]];
    for (int i = 0; i < m; ++i) {
        int i2 = (i + 1 < m) ? i + 1 : 0;
        s.n[i] = cross_vs(sub(s.v[i2], s.v[i]), 1.0f);
        normalize(s.n[i]);
    }
    s.centroid = polygon_centroid(s.v, m);
    s.meta = SHAPE_POLYGON | (m << 8);
    return true;
}

B2G_HD void build_shape(const b2g_fixture_def& d, ShapeRec& s) {
    s = ShapeRec{};
    s.radius = d.radius;
    if (d.shape_type == B2G_SHAPE_CIRCLE) {
        s.v[0] = mk(d.vertices[0].x, d.vertices[0].y);
        s.meta = SHAPE_CIRCLE | (1 << 8);
    } else if (d.shape_type == B2G_SHAPE_EDGE) {
        for (int i = 0; i < 4; ++i) s.v[i] = mk(d.vertices[i].x, d.vertices[i].y);
        s.meta = SHAPE_EDGE | (2 << 8) | ((d.one_sided ? 1 : 0) << 16);
    } else {
        if (d.polygon_mode == B2G_POLYGON_BOX) {
            polygon_box(s, d.box_half_extents.x, d.box_half_extents.y);
        } else if (d.polygon_mode == B2G_POLYGON_BOX_ORIENTED) {
            /* set_as_box_angle, b2_polygon_shape.rs:25-50 */
            polygon_box(s, d.box_half_extents.x, d.box_half_extents.y);
            Xf xf;
            xf.p = mk(d.box_center.x, d.box_center.y);
            xf.q = rot(d.box_angle);
            s.centroid = xf.p;
            for (int i = 0; i < 4; ++i) {
                s.v[i] = mul(xf, s.v[i]);
                s.n[i] = mul(xf.q, s.n[i]);
            }
        } else {
            polygon_hull(s, d.vertices, d.vertex_count);
        }
        s.radius = d.radius;
    }
}

}  // namespace b2g
#endif
