// The estimate pass's form of a scene, made at its upload (host).
#pragma once

#include <algorithm>
#include <array>
#include <cmath>
#include <tuple>
#include <vector>

#include "layout.h"
#include "scene.h"

namespace pcr {

// The estimate pass's form of the quads and spheres (device.cuh,
// flat_closest): boxes, i.e. six consecutive non-emissive quads that bound a
// rectangular box other than the room, and axis-aligned rectangles.  The
// scene takes the pass only when every quad is one of these and there are at
// most kMaxFlatPrims primitives: the pass tests them all, while past that
// number the exact tests' grouped culling skips more than it costs.
constexpr int kMaxFlatPrims = 64;
struct FlatScene {
    std::vector<DRect> rects, srects;
    std::vector<DBox> boxes;
    int n_rects[3] = {0, 0, 0}, n_inner = 0;
    float cell_lo[3] = {0, 0, 0}, cell_hi[3] = {0, 0, 0};
    bool ok = false;
    float pad = 0.f, reach = 0.f;
};
inline FlatScene flat_scene(const pcr_scene_desc& d, const std::vector<DPlane>& planes)
{
    FlatScene F;
    typedef std::array<double, 3> V;
    auto vec = [](const float* p) { return V{p[0], p[1], p[2]}; };
    auto add = [](const V& a, const V& b) { return V{a[0] + b[0], a[1] + b[1], a[2] + b[2]}; };
    auto dot = [](const V& a, const V& b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; };
    double big = 0.0;
    auto reach = [&](const V& a) { for (double x : a) big = std::max(big, std::fabs(x)); };
    reach(vec(d.cam_pos));
    for (int i = 0; i < d.n_planes; i++) {
        const V o = vec(d.planes[i].origin), u = vec(d.planes[i].u), v = vec(d.planes[i].v);
        for (const V& c : {o, add(o, u), add(o, v), add(add(o, u), v)}) reach(c);
    }
    for (int i = 0; i < d.n_spheres; i++) {
        V c = vec(d.spheres[i].center);
        for (double& x : c) x = std::fabs(x) + std::fabs(d.spheres[i].radius);
        reach(c);
    }
    if (!(big < 1e6) || d.n_planes + d.n_spheres > 6 * kMaxFlatPrims) return F;  // also NaN
    F.reach = (float)std::max(1e-2, 1.05 * big);
    F.pad = 1e-5f * F.reach;

    // six quads from i on as a box; their corners may miss the ideal ones by
    // a little (scene files round them), which goes into the box's margin
    auto as_box = [&](int i, DBox& B) {
        if (i + 6 > d.n_planes) return false;
        V n[3];
        double off[3][2];
        int slab[6], face[3][2], slabs = 0, count[3] = {0, 0, 0};
        for (int k = 0; k < 6; k++) {
            const pcr_plane& p = d.planes[i + k];
            const V m = vec(p.n), u = vec(p.u), v = vec(p.v);
            if (planes[i + k].n_emit.w != 0.f || std::fabs(dot(m, m) - 1.0) > 1e-6) return false;
            if (std::fabs(dot(u, v)) > 1e-6 * std::sqrt(dot(u, u) * dot(v, v))) return false;
            int at = 0;
            while (at < slabs && std::fabs(dot(n[at], m)) < 1.0 - 1e-10) {
                if (std::fabs(dot(n[at], m)) > 1e-6) return false;
                at++;
            }
            if (at == slabs) {
                if (slabs == 3) return false;
                n[slabs++] = m;
            }
            if (count[at] == 2) return false;
            face[at][count[at]] = i + k;
            off[at][count[at]++] = dot(n[at], vec(p.origin));
            slab[k] = at;
        }
        if (slabs != 3) return false;
        double mid[3], half[3], dev = 0.0;
        for (int a = 0; a < 3; a++) {
            mid[a] = 0.5 * (off[a][0] + off[a][1]);
            half[a] = 0.5 * std::fabs(off[a][0] - off[a][1]);
        }
        for (int k = 0; k < 6; k++) {
            const V o = vec(d.planes[i + k].origin), u = vec(d.planes[i + k].u), v = vec(d.planes[i + k].v);
            int met = 0;  // sign combinations on the two other slabs
            for (const V& c : {o, add(o, u), add(o, v), add(add(o, u), v)}) {
                int signs = 0, bit = 0;
                for (int a = 0; a < 3; a++) {
                    const double x = dot(n[a], c) - mid[a];
                    dev = std::max(dev, std::fabs(std::fabs(x) - half[a]));
                    if (a != slab[k]) signs |= (x > 0.0) << bit++;
                }
                met |= 1 << signs;
            }
            if (met != 15) return false;
        }
        if (dev > 4e-5 * F.reach) return false;
        for (int a = 0; a < 3; a++) {
            if (half[a] < 8.0 * (dev + F.pad)) return false;
            B.nc[a] = make_float4((float)n[a][0], (float)n[a][1], (float)n[a][2], (float)mid[a]);
        }
        B.h = make_float4((float)half[0], (float)half[1], (float)half[2], (float)(1.01 * dev) + F.pad);
        auto low = [&](int a) { return off[a][0] < off[a][1] ? 0 : 1; };
        B.lo = make_int4(face[0][low(0)], face[1][low(1)], face[2][low(2)], 0);
        B.hi = make_int4(face[0][1 - low(0)], face[1][1 - low(1)], face[2][1 - low(2)], 0);
        return true;
    };
    // the axis an axis-aligned rectangle is normal to, -1 for another quad
    auto rect_axis = [&](int i) {
        const pcr_plane& p = d.planes[i];
        int axis = -1, along_u = -1, along_v = -1;
        for (int k = 0; k < 3; k++) {
            const int a = (k + 1) % 3, b = (k + 2) % 3;
            if (std::fabs(p.n[k]) == 1.f && p.n[a] == 0.f && p.n[b] == 0.f) axis = k;
            if (p.u[k] != 0.f && p.u[a] == 0.f && p.u[b] == 0.f) along_u = k;
            if (p.v[k] != 0.f && p.v[a] == 0.f && p.v[b] == 0.f) along_v = k;
        }
        return along_u < 0 || along_v < 0 || along_u == along_v || along_u == axis || along_v == axis ? -1 : axis;
    };
    // Whether the box of quads i .. i + 5 is a room.  A ray that starts in a
    // box is in doubt, so a box that holds the camera or a light is none, and
    // where its quads are rectangles anyway it holds nothing else either
    // (a closed 4 x 4 x 6 room with a sphere, as a box, by the exact tests
    // alone, and as rectangles: 1 M closest hits 70, 48 and 40 us, six batched
    // renders 25.7, 22.0 and 12.4 ms).
    auto is_room = [&](int i, const DBox& B) {
        const float half[3] = {B.h.x, B.h.y, B.h.z};
        auto in = [&](const V& c) {
            for (int a = 0; a < 3; a++)
                if (!(std::fabs(dot(V{B.nc[a].x, B.nc[a].y, B.nc[a].z}, c) - B.nc[a].w) < half[a] - B.h.w)) return false;
            return true;
        };
        if (in(vec(d.cam_pos))) return true;
        bool rects = true;
        for (int k = i; k < i + 6; k++) rects = rects && rect_axis(k) >= 0;
        for (int k = 0; k < d.n_planes; k++) {
            if ((k >= i && k < i + 6) || (planes[k].n_emit.w == 0.f && !rects)) continue;
            const V o = vec(d.planes[k].origin), u = vec(d.planes[k].u), v = vec(d.planes[k].v);
            for (const V& c : {o, add(o, u), add(o, v), add(add(o, u), v)})
                if (in(c)) return true;
        }
        for (int k = 0; k < d.n_spheres && rects; k++)
            if (in(vec(d.spheres[k].center))) return true;
        return false;
    };
    // by normal axis, plane coordinate, and order in the scene
    std::vector<std::tuple<int, float, int>> flat;
    int no_box = 0;  // quads before this one are a room's
    for (int i = 0; i < d.n_planes;) {
        DBox B;
        if (i >= no_box && as_box(i, B)) {
            if (!is_room(i, B)) {
                F.boxes.push_back(B);
                i += 6;
                continue;
            }
            no_box = i + 6;
        }
        const int axis = rect_axis(i);
        if (axis < 0) return F;
        flat.push_back({axis, d.planes[i].origin[axis] + 0.f, i});  // + 0.f: -0 and +0 are one plane
        i++;
    }
    if ((int)(flat.size() + F.boxes.size()) + d.n_spheres > kMaxFlatPrims) return F;
    std::sort(flat.begin(), flat.end());
    for (size_t k = 0; k < flat.size(); k++) {
        const auto [axis, at, i] = flat[k];
        const pcr_plane& p = d.planes[i];
        const int a = axis == 0 ? 1 : 0, b = axis == 2 ? 1 : 2;  // the two other axes, in order
        auto span = [&](int x) { return (double)p.u[x] + (double)p.v[x]; };  // one of them is zero
        int flags = (planes[i].n_emit.w != 0.f ? kRectEmissive : 0) | axis << kRectAxisShift;
        if (k > 0 && std::get<0>(flat[k - 1]) == axis && std::get<1>(flat[k - 1]) == at) flags |= kRectSamePlane;
        DRect q;
        q.a = make_float4(at, (float)(p.origin[a] + 0.5 * span(a)), (float)(p.origin[b] + 0.5 * span(b)), __int_as_float_host(i));
        q.b = make_float4((float)(0.5 * std::fabs(span(a))), (float)(0.5 * std::fabs(span(b))), __int_as_float_host(flags), 0.f);
        F.rects.push_back(q);
        F.n_rects[axis]++;
    }

    // The cell: everything that is no wall, the camera included, lies in it;
    // a wall is a rectangle whose plane has all of that on one side.
    double in_lo[3], in_hi[3];
    for (int x = 0; x < 3; x++) in_lo[x] = in_hi[x] = d.cam_pos[x];
    auto hold = [&](const V& c, double r) {
        for (int x = 0; x < 3; x++) {
            in_lo[x] = std::min(in_lo[x], c[x] - r);
            in_hi[x] = std::max(in_hi[x], c[x] + r);
        }
    };
    for (const DBox& B : F.boxes)
        for (int i : {B.lo.x, B.hi.x}) {
            const V o = vec(d.planes[i].origin), u = vec(d.planes[i].u), v = vec(d.planes[i].v);
            for (const V& c : {o, add(o, u), add(o, v), add(add(o, u), v)}) hold(c, 0.0);
        }
    for (int i = 0; i < d.n_spheres; i++) hold(vec(d.spheres[i].center), std::fabs(d.spheres[i].radius));
    for (const DRect& q : F.rects)
        if (__float_as_int_host(q.b.z) & kRectEmissive) {
            const pcr_plane& p = d.planes[__float_as_int_host(q.a.w)];
            hold(vec(p.origin), 0.0);
            hold(add(vec(p.origin), add(vec(p.u), vec(p.v))), 0.0);
        }
    double lo[3], hi[3];
    for (int x = 0; x < 3; x++) { lo[x] = -HUGE_VAL; hi[x] = HUGE_VAL; }
    std::vector<DRect> walls;
    for (DRect q : F.rects) {
        const int flags = __float_as_int_host(q.b.z), x = flags >> kRectAxisShift;
        const bool above = q.a.x >= in_hi[x] - F.pad, below = q.a.x <= in_lo[x] + F.pad;
        if ((flags & kRectEmissive) || above == below) { F.srects.push_back(q); continue; }
        if (above) hi[x] = std::min(hi[x], (double)q.a.x);
        else lo[x] = std::max(lo[x], (double)q.a.x);
        walls.push_back(q);
    }
    F.n_inner = (int)F.srects.size();
    for (DRect& q : F.srects) {
        // the light's points lie in the cell, away from the walls except
        // one in its own plane, which any ray meets at the light's t
        int flags = __float_as_int_host(q.b.z);
        const int x = flags >> kRectAxisShift, y = x == 0 ? 1 : 0, z = x == 2 ? 1 : 2;
        auto clear = [&](int k, double c, double h) { return c - h > lo[k] + 4.0 * F.pad && c + h < hi[k] - 4.0 * F.pad; };
        if ((flags & kRectEmissive) && clear(y, q.a.y, q.b.x) && clear(z, q.a.z, q.b.y) &&
            (q.a.x == lo[x] || q.a.x == hi[x] || clear(x, q.a.x, 0.0)))
            flags |= kRectCellLight;
        q.b.z = __int_as_float_host(flags);
    }
    F.srects.insert(F.srects.end(), walls.begin(), walls.end());
    for (int x = 0; x < 3; x++) {
        F.cell_lo[x] = (float)(lo[x] + F.pad);
        F.cell_hi[x] = (float)(hi[x] - F.pad);
    }
    F.ok = true;
    return F;
}

}  // namespace pcr
