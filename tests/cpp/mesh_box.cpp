// mesh_may_hit against the slab test of the BVH walk: a ray that the walk
// would follow into the mesh's box may not be turned away before it, whatever
// the distance.  Prints, per distance, the rays that meet the box and how many
// of them mesh_may_hit turns away.
#include "device_on_host.h"
#include "device_host.h"

int main()
{
    using namespace pcr;
    std::mt19937_64 gen(5);
    auto uniform = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
    for (double dist : {1.0, 100.0, 1e4, 1e5, 1e6}) {
        long met = 0, lost = 0;
        for (int i = 0; i < 400000; i++) {
            const double size = i % 2 ? 0.01 : 1.0;
            float lo[3], hi[3], big = 1.f;
            double target[3], w[3], len = 0.0;
            for (int k = 0; k < 3; k++) {
                const float a = (float)uniform(-size, size), b = i % 7 == 0 && k == i % 3 ? a : (float)uniform(-size, size);
                lo[k] = std::min(a, b);
                hi[k] = std::max(a, b);
                big = std::max(big, std::max(std::fabs(a), std::fabs(b)));
                target[k] = i % 3 ? (uniform(0, 1) < 0.5 ? lo[k] : hi[k]) : uniform(lo[k], hi[k]);  // corners, inside
                w[k] = uniform(-1, 1) * (i % 5 == 0 && k == i % 3 ? 1e-4 : 1.0);
                len += w[k] * w[k];
            }
            len = std::sqrt(len);
            const float3 o = make_float3((float)(target[0] + w[0] / len * dist), (float)(target[1] + w[1] / len * dist),
                                         (float)(target[2] + w[2] / len * dist));
            double d[3] = {target[0] - o.x, target[1] - o.y, target[2] - o.z};
            const double l = std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
            const float3 dir = make_float3((float)(d[0] / l), (float)(d[1] / l), (float)(d[2] / l));
            const float3 inv = make_float3(__fdiv_rn(1.f, dir.x), __fdiv_rn(1.f, dir.y), __fdiv_rn(1.f, dir.z));
            DScene S;
            std::memset((void*)&S, 0, sizeof S);
            S.n_nodes = 1;
            const float pad = 1e-4f * big;  // as the scene upload pads it
            S.mesh_lo = make_float4(lo[0] - pad, lo[1] - pad, lo[2] - pad, 0.f);
            S.mesh_hi = make_float4(hi[0] + pad, hi[1] + pad, hi[2] + pad, 0.f);
            if (slab4(lo[0], hi[0], lo[1], hi[1], lo[2], hi[2], o, inv, FLT_MAX) > FLT_MAX) continue;
            met++;
            if (!mesh_may_hit(S, o, dir, FLT_MAX)) lost++;
        }
        std::printf("%g %ld %ld\n", dist, met, lost);
    }
}
