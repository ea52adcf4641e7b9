// Test-only library: the choice between the wide BVH and the BVH2 that the ray-query kernels make for
// each ray (pt_scene.cuh wide_ray), and both traversals, compiled for the host.  Built by
// tests/test_wide_ray_host.py; never part of the product.
#include <vector>

#include "../../open_rendering_framework_b200/csrc/pt_bvh.h"
#include "../../open_rendering_framework_b200/csrc/pt_scene.cuh"

using namespace pt;

struct QueryScene {
  BvhHost bvh;
  std::vector<float4> nodes4;
  SceneDev S;
};

extern "C" __attribute__((visibility("default"))) void* hq_build(const float* tri_pos, unsigned n)
{
  QueryScene* h = new QueryScene();
  int depth4 = 0;
  if (!build_bvh(tri_pos, n, h->bvh) || !build_bvh4(h->bvh, h->nodes4, depth4, BvhParams())) {
    delete h;
    return nullptr;
  }
  memset(&h->S, 0, sizeof(h->S));
  h->S.nodes = h->bvh.nodes.data();
  h->S.tri_v0 = h->bvh.tri_v0.data();
  h->S.tri_e1 = h->bvh.tri_e1.data();
  h->S.tri_e2 = h->bvh.tri_e2.data();
  h->S.n_tris = n;
  h->S.nodes4 = h->nodes4.data();
  h->S.trav_scale = scene_diagonal(tri_pos, n, &h->S.trav_reach);
  return h;
}
extern "C" __attribute__((visibility("default"))) unsigned long long hq_bary_at(unsigned i) { return bary_at(i); }
extern "C" __attribute__((visibility("default"))) unsigned hq_rays_per_warp(unsigned n, unsigned warps) { return rays_per_warp(n, warps); }
extern "C" __attribute__((visibility("default"))) void hq_free(void* h) { delete (QueryScene*)h; }
// rays: n x 8 floats (origin, tmin, direction, tmax).  wide: whether the ray is traced over the wide BVH;
// prim / t / any and prim2 / t2 / any2: the results over the wide BVH (where wide) and over the BVH2.
extern "C" __attribute__((visibility("default"))) void hq_trace(void* hp, const float* rays, long n, int* wide, int* prim, float* t, int* any,
                                                                int* prim2, float* t2, int* any2)
{
  QueryScene* h = (QueryScene*)hp;
  const TravGeom g = trav_geom(h->S);
  for (long i = 0; i < n; ++i) {
    const float* r = rays + 8 * i;
    const float3 o = make_float3(r[0], r[1], r[2]), d = make_float3(r[4], r[5], r[6]);
    Hit hh = trace_closest(g, o, d, r[3], r[7]);
    prim2[i] = hh.prim;
    t2[i] = hh.prim >= 0 ? hh.t : -1.0f;
    any2[i] = trace_any(g, o, d, r[3], r[7]) ? 1 : 0;
    wide[i] = wide_ray(o, d, r[3], g) ? 1 : 0;
    prim[i] = prim2[i];
    t[i] = t2[i];
    any[i] = any2[i];
    if (!wide[i]) continue;
    uint2 ring[kRing4], spill[kSpill4];
    Stack4 s4;
    stack4_init(s4, ring, 1, spill);
    const RayPre4 rp = ray_pre4(o, d, g.trav_scale);
    hh.t = r[7];
    hh.u = hh.v = 0.0f;
    hh.prim = -1;
    for (int cur = 0; cur != kDone4;) {
      if (cur < 0) {
        leaf_closest(g, (uint32_t)cur, o, d, r[3], hh);
        cur = stack4_next(s4, hh.t, true);
      } else {
        cur = trav4_node_closest(g, cur, rp, r[3], hh, s4);
      }
    }
    prim[i] = hh.prim;
    t[i] = hh.prim >= 0 ? hh.t : -1.0f;
    any[i] = trace_any_wide(g, o, d, r[3], r[7]) ? 1 : 0;
  }
}
