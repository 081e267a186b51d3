// Which rays of a scene the estimate pass leaves to the exact tests, and
// whether its answers are theirs.  One line per scene: name, whether the pass
// takes the scene, its rectangles, its boxes, rays, closest-hit rays in doubt,
// wrong answers, shadow rays in doubt, wrong answers.
#include "device_on_host.h"
#include "device_host.h"
#include "flat_scene.h"

using namespace pcr;

struct Room {
    std::vector<pcr_plane> quads;
    std::vector<pcr_sphere> spheres;
    float cam[3] = {0.f, 0.f, -0.5f};
    double turn = 0.0;  // about y, around (0, 0, -3)

    void quad(std::array<double, 3> o, std::array<double, 3> u, std::array<double, 3> v, int mat = 0)
    {
        const double c = std::cos(turn), s = std::sin(turn);
        auto rot = [&](std::array<double, 3> a) { return std::array<double, 3>{c * a[0] + s * a[2], a[1], c * a[2] - s * a[0]}; };
        o[2] += 3.0;
        o = rot(o);
        o[2] -= 3.0;
        u = rot(u);
        v = rot(v);
        pcr_plane p{};
        const double n[3] = {u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]};
        const double l = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        for (int k = 0; k < 3; k++) {
            p.origin[k] = (float)o[k];
            p.u[k] = (float)u[k];
            p.v[k] = (float)v[k];
            p.n[k] = (float)(n[k] / l);
        }
        p.area = (float)l;
        p.mat = mat;
        quads.push_back(p);
    }
    void box(std::array<double, 3> lo, std::array<double, 3> size)
    {
        for (int a = 0; a < 3; a++) {
            std::array<double, 3> u{0, 0, 0}, v{0, 0, 0}, far = lo;
            u[(a + 1) % 3] = size[(a + 1) % 3];
            v[(a + 2) % 3] = size[(a + 2) % 3];
            far[a] += size[a];
            quad(lo, u, v);
            quad(far, u, v);
        }
    }
    void sphere(double x, double y, double z, double r) { spheres.push_back({{(float)x, (float)y, (float)z}, (float)r, 0}); }

    void measure(const char* name)
    {
        const int n_planes = (int)quads.size();
        std::vector<DPlane> planes(n_planes), dark;
        std::vector<float4> groups, dark_groups;
        std::vector<DSphere> balls;
        DScene S;
        std::memset((void*)&S, 0, sizeof S);
        auto square = [](const float* a) { return __fadd_rn(__fadd_rn(__fmul_rn(a[0], a[0]), __fmul_rn(a[1], a[1])), __fmul_rn(a[2], a[2])); };
        auto alone = [](std::vector<float4>& g, int i) {
            g.push_back(make_float4(0.f, 0.f, 0.f, __int_as_float(i)));
            g.push_back(make_float4(0.f, 0.f, 0.f, __int_as_float(1)));
        };
        for (int i = 0; i < n_planes; i++) {
            const pcr_plane& p = quads[i];
            planes[i].o_mat = make_float4(p.origin[0], p.origin[1], p.origin[2], __int_as_float(p.mat));
            planes[i].n_emit = make_float4(p.n[0], p.n[1], p.n[2], p.mat ? 1.f : 0.f);
            planes[i].u_uu = make_float4(p.u[0], p.u[1], p.u[2], square(p.u));
            planes[i].v_vv = make_float4(p.v[0], p.v[1], p.v[2], square(p.v));
            alone(groups, i);
            if (p.mat) S.emit_planes[S.n_emit_planes++] = i;
            else { alone(dark_groups, (int)dark.size()); dark.push_back(planes[i]); }
        }
        for (const pcr_sphere& s : spheres) {
            DSphere b;
            b.c_r = make_float4(s.center[0], s.center[1], s.center[2], s.radius);
            b.mat = make_int4(0, 0, 0, 0);
            balls.push_back(b);
        }
        pcr_scene_desc d{};
        d.n_planes = n_planes;
        d.planes = quads.data();
        d.n_spheres = (int)spheres.size();
        d.spheres = spheres.data();
        std::copy(cam, cam + 3, d.cam_pos);
        const FlatScene F = flat_scene(d, planes);
        S.planes = planes.data();
        S.n_planes = n_planes;
        S.spheres = balls.data();
        S.n_spheres = (int)balls.size();
        S.pgroups = groups.data();
        S.n_pgroups = n_planes;
        S.splanes = dark.data();
        S.sgroups = dark_groups.data();
        S.n_sgroups = (int)dark.size();
        S.rects = F.rects.data();
        S.boxes = F.boxes.data();
        S.n_boxes = (int)F.boxes.size();
        S.srects = F.srects.data();
        S.n_srects = (int)F.srects.size();
        S.n_inner = F.n_inner;
        for (int k = 0; k < 3; k++) {
            S.n_rects[k] = F.n_rects[k];
            S.cell_lo[k] = F.cell_lo[k];
            S.cell_hi[k] = F.cell_hi[k];
        }
        S.flat_ok = F.ok;
        S.flat_pad = F.pad;
        S.flat_reach = F.reach;
        DMaterial mats[2] = {};
        mats[1].flags = kMatEmissive;

        std::mt19937_64 gen(9);
        auto uniform = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
        std::normal_distribution<double> normal;
        const int n = 200000;
        int doubt = 0, wrong = 0, s_doubt = 0, s_wrong = 0;
        const pcr_plane& light = quads[0];
        for (int i = 0; i < n; i++) {
            float3 o = make_float3((float)uniform(-1.9, 1.9), (float)uniform(-1.9, 1.9), (float)uniform(-5.9, -0.1));
            double v[3] = {normal(gen), normal(gen), normal(gen)};
            const double l = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
            const float3 dir = make_float3((float)(v[0] / l), (float)(v[1] / l), (float)(v[2] / l));
            float t = FLT_MAX, exact_t = FLT_MAX;
            uint32_t prim = 0;
            const uint32_t exact = scene_analytic_exact(S, o, dir, exact_t);
            if (!F.ok || !flat_closest(S, o, dir, t, prim)) doubt++;
            else if (prim != exact || t != exact_t) wrong++;
            const double a = uniform(0, 1), b = uniform(0, 1);
            const float3 to = make_float3((float)(light.origin[0] + a * light.u[0] + b * light.v[0]) - o.x,
                                          (float)(light.origin[1] + a * light.u[1] + b * light.v[1]) - o.y,
                                          (float)(light.origin[2] + a * light.u[2] + b * light.v[2]) - o.z);
            const float d2 = f3dot(to, to);
            const float3 wi = f3mul(to, rsqrtf(d2));
            float bound;
            int at;
            const int query = F.ok ? flat_blocked(S, o, wi, d2, at) : -1;
            if (query < 0) s_doubt++;
            else if (query != scene_blocked_exact<false>(S, mats, o, wi, shadow_end(d2), (double)d2 - 1e-3, bound)) s_wrong++;
        }
        std::printf("%s %d %zu %zu %d %d %d %d %d\n", name, (int)F.ok, F.rects.size(), F.boxes.size(), n, doubt, wrong, s_doubt, s_wrong);
    }
};

static Room lit_room(double light_y)
{
    Room r;
    r.quad({-0.5, light_y, -4}, {1, 0, 0}, {0, 0, 1}, 1);
    return r;
}

int main()
{
    { Room r = lit_room(1.99); r.box({-2, -2, -6}, {4, 4, 6}); r.sphere(0.5, -1.4, -3, 0.6); r.measure("closed"); }
    { Room r = lit_room(2.0); r.box({-2, -2, -6}, {4, 4, 6}); r.box({-1, -2, -4}, {1, 1.5, 1}); r.measure("closed-furnished"); }
    // the camera outside: the light and the sphere still make it a room
    { Room r = lit_room(1.99); r.box({-2, -2, -6}, {4, 4, 6}); r.cam[2] = 9.f; r.sphere(0.5, -1.4, -3, 0.6); r.measure("closed-seen-from-outside"); }
    // a box that holds nothing stays one; so does one with a light lying on it
    { Room r = lit_room(1.99); r.box({-1, -2, -4}, {1, 1.5, 1}); r.measure("box"); }
    { Room r = lit_room(-0.5); r.box({-0.7, -2, -4.2}, {1.4, 1.5, 1.4}); r.measure("lit-box"); }
    // turned, its walls are no rectangles: the scene takes the exact tests
    { Room r = lit_room(1.99); r.turn = 0.3; r.box({-4, -2, -8}, {8, 4, 10}); r.measure("closed-turned"); }
}
