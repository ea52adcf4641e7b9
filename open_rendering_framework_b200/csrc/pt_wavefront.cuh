// The wavefront's device state and the vertices of a path: one function per material class, following the
// reference's material programs, on the per-path records.  The wavefront's shading kernels (pt_render.cu)
// and the path pools (pt_pool.cuh) run the same functions, so both give a path the same arithmetic.
#pragma once
#include <utility>
#include <vector>

#include "pt_context.h"

namespace pt {

constexpr int kBlock = 128;
constexpr int kWarps = kBlock / 32;
// The 4-wide persistent kernels alternate warp-wide phases of leaf tests and node steps.  Closest hit:
// a leaf phase once the lanes holding a leaf are at least twice those that can take a node step
// (leaf tests wait for more company); any hit: once they are at least half of them (an occluder found
// early ends the ray).  Measured against "at least as many" on the single-scene render: +0.5 %.
constexpr int kLeafVsNodeClosest = 2;
constexpr int kLeafVsNodeAny = 2;

// Per-path metadata in rng.w
constexpr uint32_t META_DEPTH = 0xffffu;
constexpr uint32_t META_EMIT = 1u << 16;
constexpr uint32_t META_OUTSIDE = 1u << 17;
constexpr uint32_t META_PROBE = 1u << 18;  // a probe's indirect path (sample_camera.cu:168-206)
constexpr int META_GSHIFT = 24;            // pending dipole gathers on the path's stack (8 bits)
constexpr uint32_t META_KEEP = ~(META_DEPTH | META_EMIT);

// One 16-byte field of a per-path pair record: field k of path i sits at rec[2 i + k].  The ray (origin,
// direction) and the path state (throughput, rng state) are two 32-byte records per path, each one
// whole sector: a shading kernel reading and rewriting a path at a random id touches two whole sectors
// instead of four half sectors of four arrays, and the extend kernel reads exactly the ray's sector
// (consecutive paths' rays are contiguous).
template <class T> struct Field2 {
  T* p;
  __device__ __forceinline__ T& operator[](uint64_t i) const { return p[2 * i]; }
};

struct WfDev {
  Field2<float4> ray_o;
  Field2<float4> ray_d;
  Field2<float4> thr;
  float4* rad;
  Field2<uint4> rng;
  float4* hit;
  uint32_t* q_in;
  uint32_t* q_out;
  uint32_t* q_mat;  // kQueues * cap
  uint8_t* cls_of;  // material class of the ray at each position of q_in (written by extend, binned by k_bin_*)
  uint32_t* bin;    // per chunk of kBinChunk queue positions: kQueues class counts, then starts in the queues
  float4* sh_o;
  float4* sh_d;
  float4* sh_c;
  uint32_t* sh_pid;
  uint32_t* cnt;
  uint64_t cap;
  int in_slot, out_slot;
  // pending dipole gathers, [slot * cap + path]: (xo, throughput.x), (no, throughput.y), (throughput.z, material)
  float4* g_a;
  float4* g_b;
  float2* g_c;
  float4* g_d;  // the gather's weight (rough boundary) and 1, or (1, 1, 1, 0) for a smooth boundary
  uint32_t g_slots;
  // adjoint renders: per path (image gradient of the path, pending kind) and (pending d w / w, index)
  float4* adj_a;
  float4* adj_b;
  // the scenes and items of the pass; each path's item
  const SceneDev* scenes;
  const ItemDev* items;
  uint32_t n_items;
  uint32_t multi;   // 0: every path of the chunk renders scenes[scene0]
  uint32_t scene0;
  uint16_t* path_item;
};

// Probe storage of a pass, indexed by probe id (item after item, then frame, object, sample).
struct SssDev {
  float4* probes;      // 5 float4 per PositionSample
  float4* pc_pos;      // compacted probes with L != 0 per (frame, object) set, at the set's first probe id: pos
  float4* pc_wl;       //   weight * L
  float4* pc_nrm;      //   normal
  float4* pc_tr;       //   transmitted
  uint32_t* pc_cnt;    //   count per set
};

// Index of the last item whose begin field is <= key (every begin field increases item after item).
template <class F>
__device__ __forceinline__ uint32_t find_item(const ItemDev* items, uint32_t n, uint64_t key, F begin)
{
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if ((uint64_t)begin(items[mid]) <= key) lo = mid;
    else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ const SceneDev& scene_of(const WfDev& w, uint32_t pid)
{
  const uint32_t k = w.multi ? w.items[w.path_item[pid]].scene : w.scene0;
  return w.scenes[k];
}

__device__ __forceinline__ unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }
__device__ __forceinline__ unsigned long long* cnt64(uint32_t* cnt, int slot) { return reinterpret_cast<unsigned long long*>(cnt + slot); }

// Block-aggregated append: every thread of the block calls this (uniform control flow); threads
// with want == true receive a distinct slot in [0, *counter).  One global atomic per block.
__device__ __forceinline__ uint32_t block_slot(bool want, uint32_t* counter, uint32_t* smem /* kWarps + 1 */)
{
  unsigned m = __ballot_sync(0xffffffffu, want);
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) smem[warp] = __popc(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t total = 0;
    for (int w = 0; w < kWarps; ++w) {
      uint32_t c = smem[w];
      smem[w] = total;
      total += c;
    }
    smem[kWarps] = total ? atomicAdd(counter, total) : 0u;
  }
  __syncthreads();
  uint32_t slot = smem[kWarps] + smem[warp] + __popc(m & lanemask_lt());
  __syncthreads();
  return slot;
}


// Shading normal of a hit: normalize(rtTransformNormal(normalize(n))) with the identity transform,
// where n is the interpolated vertex normal or the geometric normal (triangle_mesh.cu:63-70,
// diffuse_shader.cu:48).
__device__ __forceinline__ float3 shading_normal(const SceneDev& S, const int4& info, float u, float v, int prim)
{
  float3 n;
  if (info.x >= 0) {
    float3 n0 = ld3(__ldg(S.normals + info.x)), n1 = ld3(__ldg(S.normals + info.y)), n2 = ld3(__ldg(S.normals + info.z));
    n = normalize(n1 * u + n2 * v + n0 * (1.0f - u - v));
  } else {
    n = normalize(ld3(__ldg(S.geo + prim)));
  }
  return normalize(n);
}

// Visibility for the vertex programs that trace a shadow ray of their own (one copy, out of line).  Over
// the wide BVH where its box tests hold, as the shadow kernels: a third less for a pass of layered objects with
// the multiple-scattering model than over the BVH2.
static __device__ __noinline__ bool occluded(const SceneDev& S, float3 o, float3 d, float tmin, float tmax)
{
  const TravGeom g = trav_geom(S);
  const bool hit = g.nodes4 && wide_ray(o, d, tmin, g) ? trace_any_wide(g, o, d, tmin, tmax) : trace_any(g, o, d, tmin, tmax);
  return hit || (S.n_ana && ana_any(S, o, d, tmin, tmax));
}

// ------------------------------------------------------------------ lights (LightSampler.h)
__device__ __forceinline__ float3 ldf3(const float* p) { return f3(p[0], p[1], p[2]); }

// evaluate_direct_illumination, LightSampler.h:143-166 (all five light types).  Out-of-range
// triangle indices (a draw that rounds to 1.0) are clamped and counted.
static __device__ void eval_direct(const SceneDev& S, const float3& pos, const LightRaw& ls, float3& dir, float3& L, float& dist, uint32_t& seed,
                            uint32_t& clamped)
{
  const float3 em = ldf3(ls.emitted);
  switch (ls.type) {
    case POINT_LIGHT: {  // :20-28
      dir = ldf3(ls.p) - pos;
      float r2 = dot(dir, dir);
      dist = sqrtf(r2);
      dir = dir / dist;
      L = em / r2;
      break;
    }
    case DIRECTIONAL_LIGHT: {  // :31-37
      dir = normalize(-ldf3(ls.p));
      dist = kDefaultMax;
      L = em;
      break;
    }
    case TRIANGLES_AREA_LIGHT: {  // :40-71
      float cnt_f = ls.p[0], start_f = ls.p[1];
      uint32_t tris = (uint32_t)cnt_f;
      uint32_t tid = (uint32_t)((float)(uint32_t)(rnd_tea(seed) * (float)tris) + start_f);
      if (tid >= (uint32_t)S.n_tri_lights) { tid = (uint32_t)S.n_tri_lights - 1; ++clamped; }
      const TriLightRaw& tl = S.tri_lights[tid];
      float3 uvw = sample_barycentric(seed);
      float3 v0 = ldf3(tl.v0), v1 = ldf3(tl.v1), v2 = ldf3(tl.v2);
      float3 lp = v0 * uvw.x + v1 * uvw.y + v2 * uvw.z;
      float3 n = tl.has_normals ? normalize(ldf3(tl.n0) * uvw.x + ldf3(tl.n1) * uvw.y + ldf3(tl.n2) * uvw.z) : normalize(cross(v1 - v0, v2 - v0));
      dir = lp - pos;
      float sq = dot(dir, dir);
      dist = sqrtf(sq);
      dir = normalize(dir);
      float cp = fmaxf(dot(n, -dir), 0.0f);
      L = em * (tl.area * cp / sq * (float)tris);
      break;
    }
    case DISK_LIGHT: {  // :73-101
      float3 lp = ldf3(ls.p);
      float radius = ls.pad[0];
      float theta = ls.pad[2] * kPi / 180.0f, phi = ls.pad[1] * kPi / 180.0f;
      float area = kPi * radius * radius;
      float pdf = 1.0f / area;
      float3 nrm = f3(sinf(theta) * sinf(phi), cosf(theta), sinf(theta) * cosf(phi));
      float3 U, V;
      create_onb(nrm, U, V);
      float u1 = rnd_tea(seed), u2 = rnd_tea(seed);
      float r = sqrtf(u1) * radius;
      float t = 2.0f * kPi * u2;
      float3 dp = f3(r * cosf(t), r * sinf(t), 0.0f);
      dp = dp.x * U + dp.y * V + dp.z * nrm;
      lp = lp + dp;
      dir = lp - pos;
      float sq = dot(dir, dir);
      dist = sqrtf(sq);
      dir = normalize(dir);
      float cp = fmaxf(dot(nrm, -dir), 0.0f);
      L = em * (cp / sq) / pdf;
      break;
    }
    case SPHERICAL_LIGHT: {  // :103-141
      float3 lp = ldf3(ls.p);
      float radius = ls.pad[0];
      float3 vn = normalize(pos - lp);
      float3 U, V;
      create_onb(vn, U, V);
      float area = 4.0f * kPi * radius * radius;
      float pdf = 1.0f / area;
      float u1 = rnd_tea(seed), u2 = rnd_tea(seed);
      float z = u1;
      float3 sp = radius * f3(cosf(2.0f * kPi * u2) * sqrtf(1.0f - z * z), sinf(2.0f * kPi * u2) * sqrtf(1.0f - z * z), z);
      sp = sp.x * U + sp.y * V + sp.z * vn + lp;
      float3 nrm = normalize(sp - lp);
      dir = sp - pos;
      float sq = dot(dir, dir);
      dist = sqrtf(sq);
      dir = normalize(dir);
      float cp = fmaxf(dot(nrm, -dir), 0.0f);
      L = em * (cp / sq) / pdf;
      break;
    }
    case ENVMAP_LIGHT: {  // the environment map as a light: sample_environment (Envmap.h:66-98)
      sample_environment(S.env, dir, L, seed);
      dist = kDefaultMax;
      break;
    }
    default:
      dir = f3s(0.0f);
      L = f3s(0.0f);
      dist = 0.0f;
      break;
  }
}


// ------------------------------------------------------------------ MD5 stream across vertices
// The diffuse, conductor, rough-dielectric and layered shaders hand their child ray only the tea seed
// (diffuse_shader.cu:92-101, metallic_shader.cu:76-156, rough_transparent_shader.cu:114-220,
// lambertian_interface_shader.cu:143-147, rough_diffuse_shader.cu:207-211): their own
// MD5 state is never updated from the child, so after such a vertex returns, the dipole gathers of the
// translucent vertices above it draw from the MD5 state the vertex was entered with (the oracle passes
// that state down to the child, which the reference leaves uninitialised).  The wavefront keeps one
// running MD5 state per path and evaluates the gathers at the end, newest first; a vertex of those
// shaders with gathers pending above it therefore pushes a reset marker holding its entry state,
// which the gather evaluation restores when it reaches the marker.  The smooth transparent shader
// traces its child with its own payload (transparent_shader.cu:110-112), so the MD5 state simply
// runs on through it and it pushes no marker.
__device__ __forceinline__ uint32_t push_md5_reset(const WfDev& w, uint32_t pid, uint32_t meta, uint32_t s64x, uint32_t s64y, uint32_t& overflow)
{
  if (!(meta & META_PROBE) && (meta >> META_GSHIFT) != 0) {
    const uint32_t slot = meta >> META_GSHIFT;
    if (slot < w.g_slots) {
      size_t at = (size_t)slot * w.cap + pid;
      w.g_a[at] = make_float4(__uint_as_float(s64x), __uint_as_float(s64y), 0.0f, 0.0f);
      w.g_b[at] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      w.g_c[at] = make_float2(0.0f, __int_as_float(-1));
      meta += 1u << META_GSHIFT;
    } else {
      ++overflow;
    }
  }
  return meta;
}

// ------------------------------------------------------------------ path replay backprop
// The adjoint render replays every camera path with the same random numbers (same kernels, same
// decisions) and differentiates the path's contribution with respect to the scene parameters,
// with sampling detached: directions, Russian-roulette and acceptance decisions and their
// probabilities are those of the forward render; only the weights and emissions that the parameters
// enter are differentiated (M. Vicini, S. Speierer, W. Jakob, "Path replay backpropagation",
// SIGGRAPH 2021).  With T_k the throughput at vertex k, w_k its weight and E_k what vertex k adds
// to the path radiance L = sum_k T_k E_k:
//   dL/dtheta = sum_k T_k dE_k/dtheta + (dw_k/dtheta / w_k) R_{k+1},   R_{k+1} = sum_{m>k} T_m E_m.
// R starts as the forward render's L of the path and loses T_k E_k as the replay passes vertex k, so
// nothing of the path is stored: a vertex leaves (dw/w, parameter) pending in the path state, and the
// next kernel that handles the path -- after the shadow ray of the vertex has been resolved -- adds it
// times the current R.  Each gradient is weighted by the path's image gradient dLoss/dL.
enum PendingKind : uint32_t { PEND_NONE = 0, PEND_ALBEDO = 1, PEND_ROUGH = 2, PEND_SIGMA = 3 };
constexpr uint32_t kNoTexel = 0xffffffffu;

__device__ __forceinline__ void set_pending(const WfDev& w, uint32_t pid, uint32_t kind, uint32_t id, uint32_t index, const float3& d)
{
  float4 a = w.adj_a[pid];
  w.adj_a[pid] = make_float4(a.x, a.y, a.z, __uint_as_float(kind | (id << 8)));
  w.adj_b[pid] = make_float4(d.x, d.y, d.z, __uint_as_float(index));
}

// Adds the pending gradient of the path's previous vertex (R is the radiance collected beyond it).
__device__ __forceinline__ void apply_pending(const SceneDev& S, const WfDev& w, uint32_t pid)
{
  float4 a = w.adj_a[pid];
  const uint32_t kind = __float_as_uint(a.w);
  if ((kind & 0xffu) == PEND_NONE) return;
  const float4 b = w.adj_b[pid];
  const float3 R = ld3(w.rad[pid]);
  const uint32_t id = kind >> 8, idx = __float_as_uint(b.w);
  switch (kind & 0xffu) {
    case PEND_ALBEDO: {
      float* g = S.tex[id].grad;
      if (g) {
        atomicAdd(g + 3 * idx, a.x * b.x * R.x);
        atomicAdd(g + 3 * idx + 1, a.y * b.y * R.y);
        atomicAdd(g + 3 * idx + 2, a.z * b.z * R.z);
      }
      break;
    }
    case PEND_ROUGH: {
      float* g = S.tex[id].grad;
      if (g) atomicAdd(g + idx, (a.x * R.x + a.y * R.y + a.z * R.z) * b.x);
      break;
    }
    case PEND_SIGMA: {
      float* g = S.mat_grad[id];
      if (g) {
        // b = d w / d sigma_a / w per channel; sigma_s' enters the extinction divided by (1 - g)
        // (standard dipole) or times (1 + g) (delta-Eddington, directional dipole)
        const float3 mc = S.scat[id].meancosine;
        const bool dir = S.mats[id].model == DIRECTIONAL_DIPOLE;
        const float3 k = dir ? f3(1.0f + mc.x, 1.0f + mc.y, 1.0f + mc.z) : f3(1.0f / (1.0f - mc.x), 1.0f / (1.0f - mc.y), 1.0f / (1.0f - mc.z));
        const float3 ga = f3(a.x * b.x * R.x, a.y * b.y * R.y, a.z * b.z * R.z);
        atomicAdd(g + 0, ga.x);
        atomicAdd(g + 1, ga.y);
        atomicAdd(g + 2, ga.z);
        atomicAdd(g + 3, ga.x * k.x);
        atomicAdd(g + 4, ga.y * k.y);
        atomicAdd(g + 5, ga.z * k.z);
      }
      break;
    }
    default:
      break;
  }
  w.adj_a[pid] = make_float4(a.x, a.y, a.z, __uint_as_float(PEND_NONE));
}

// d ln D / d alpha of the GGX distribution at microfacet normal m (ggx_distribution):
// D = alpha^2 / (pi cos^4 (alpha^2 + tan^2)^2).
__device__ __forceinline__ float ggx_dlnD(const float3& m, const float3& n, float alpha)
{
  float c = dot(m, n);
  if (!(c > 0.0f)) return 0.0f;
  float c2 = c * c, t2 = (1.0f - c2) / c2, a2 = alpha * alpha;
  return 2.0f / alpha - 4.0f * alpha / (a2 + t2);
}
// d ln G1 / d alpha of the GGX Smith masking (ggx_G1_cos): G1 = 2 / (1 + sqrt(1 + alpha^2 tan^2)).
__device__ __forceinline__ float ggx_dlnG1(const float3& v, const float3& n, float alpha)
{
  float c = dot(v, n);
  float c2 = c * c, t2 = (1.0f - c2) / c2;
  float q = sqrtf(1.0f + alpha * alpha * t2);
  return -(alpha * t2 / q) / (1.0f + q);
}


__device__ __forceinline__ int class_of(uint32_t type)
{
  switch (type) {
    case MAT_DIFFUSE: return QC_DIFFUSE;
    case MAT_LAMBERTIAN_INTERFACE: return QC_LAYERED;
    case MAT_ROUGH_DIFFUSE: return QC_LAYERED;
    case MAT_METAL: return QC_METAL;
    case MAT_ROUGH_GLASS: return QC_GLASS;
    case MAT_TRANSPARENT: return QC_GLASS;
    case MAT_TRANSLUCENT: return QC_TRANS;
    case MAT_ROUGH_TRANSLUCENT: return QC_TRANS;
    case MAT_LIGHT: return QC_LIGHT;
    default: return -1;
  }
}

// Adds an unoccluded next-event estimate to the path (kAdj: takes it off R, and adds the albedo
// texel's gradient: the estimate is linear in the albedo).
template <bool kAdj>
__device__ __forceinline__ void shadow_unoccluded(const SceneDev& S, const WfDev& w, uint32_t slot, uint32_t p)
{
  const float4 c = w.sh_c[slot], r = w.rad[p];
  if constexpr (kAdj) {
    w.rad[p] = make_float4(r.x - c.x, r.y - c.y, r.z - c.z, 0.0f);
    const uint32_t code = __float_as_uint(c.w);
    if (code != kNoTexel) {
      const TexDev& T = S.tex[code >> 24];
      const uint32_t tx = code & 0xffffffu;
      if (T.grad) {
        const float4 a = w.adj_a[p];
        atomicAdd(T.grad + 3 * tx, a.x * c.x / __ldg(T.data + 3 * tx));
        atomicAdd(T.grad + 3 * tx + 1, a.y * c.y / __ldg(T.data + 3 * tx + 1));
        atomicAdd(T.grad + 3 * tx + 2, a.z * c.z / __ldg(T.data + 3 * tx + 2));
      }
    }
  } else {
    w.rad[p] = make_float4(r.x + c.x, r.y + c.y, r.z + c.z, 0.0f);
  }
}

// The shadow ray of a next-event estimate and what it adds to the path when nothing is in the way.
struct NeeRay {
  float3 o, d, c;
  float tmax = 0.0f, eps = 0.0f;
  uint32_t texel = kNoTexel;  // the albedo texel the estimate is linear in (adjoint), or none
};
__device__ __forceinline__ void put_nee(const WfDev& w, uint32_t at, const NeeRay& r)
{
  w.sh_o[at] = make_float4(r.o.x, r.o.y, r.o.z, r.eps);
  w.sh_d[at] = make_float4(r.d.x, r.d.y, r.d.z, r.tmax);
  w.sh_c[at] = make_float4(r.c.x, r.c.y, r.c.z, __uint_as_float(r.texel));
}

// constantbg.cu:16-19 / envmap_background.cu:20-23.  With the environment map registered as a light,
// a miss after next-event estimation (emission disabled) adds nothing, as for area lights.
// kAdj (all shade kernels): the adjoint replay; the first thing done for a path is adding the pending
// gradient of its previous vertex, and what the forward adds to the path radiance is taken off R.
template <bool kAdj>
__device__ __forceinline__ void miss_path(const SceneDev& S, const WfDev& w, uint32_t pid)
{
  if constexpr (kAdj) apply_pending(S, w, pid);
  float3 bg = S.bg_color;
  if (S.env.present) {
    if (S.env.is_light && !(w.rng[pid].w & META_EMIT)) return;
    bg = env_lookup(S.env, ld3(w.ray_d[pid]));
  }
  float4 t = w.thr[pid], r = w.rad[pid];
  float3 L = kAdj ? ld3(r) - ld3(t) * bg : ld3(r) + ld3(t) * bg;
  w.rad[pid] = make_float4(L.x, L.y, L.z, 0.0f);
}

// arealight_shader.cu:36-50: emitted radiance if the hit is front-facing and emission is enabled.
template <bool kAdj>
__device__ __forceinline__ void light_path(const SceneDev& S, const WfDev& w, uint32_t pid)
{
  if constexpr (kAdj) apply_pending(S, w, pid);
  if (!(w.rng[pid].w & META_EMIT)) return;
  float4 h = w.hit[pid], d = w.ray_d[pid];
  int prim = __float_as_int(h.w);
  float3 normal, Le;
  if ((uint32_t)prim >= S.n_tris) {  // a disk or sphere light's geometry with the same emitter program
    const uint32_t k = (uint32_t)prim - S.n_tris;
    normal = ana_normal(S, k, ld3(w.ray_o[pid]), ld3(d), h.x);
    Le = ld3(__ldg(S.ana + 3 * k + 2));
  } else {
    int4 info = __ldg(S.tri_info + prim);
    normal = shading_normal(S, info, h.y, h.z, prim);
    const MatDev& m = S.mats[info.w];
    Le = f3(m.a.x, m.a.y, m.a.z);
  }
  if (dot(normal, -ld3(d)) > 0.0f) {
    float4 t = w.thr[pid], r = w.rad[pid];
    float3 L = kAdj ? ld3(r) - ld3(t) * Le : ld3(r) + ld3(t) * Le;
    w.rad[pid] = make_float4(L.x, L.y, L.z, 0.0f);
  }
}

// rough_diffuse_shader.cu:55-292, one vertex of a Lambertian base under a rough dielectric interface:
// a visible microfacet normal from two tea draws and its Fresnel reflectance R_i; a light sample whose
// shadow ray is traced here, because the reference evaluates the multiscattering BSDFs (which draw tea
// randoms) and clears emit_light only when the light is visible; then, with probability 1 - R_i, the
// base (cosine-weighted about the microfacet normal, or the multiscattering diffuse walk) and otherwise
// the mirror reflection about the microfacet normal (or the multiscattering conductor walk with
// eta = 1 / ior, whose weight the reference does not apply).  Adds the light estimate to the path
// radiance, writes the continuation ray and throughput, and returns whether the path continues.
__device__ __forceinline__ bool rough_diffuse_vertex(const SceneDev& S, const WfDev& w, uint32_t pid, const float3& hit_pos, const float3& d,
                                                  const float3& normal, const float3& ffnormal, const MatDev& m, uint32_t& t, bool& emit,
                                                  uint32_t& clamped, int& capped)
{
  const float3 w_i = -d;
  const float3 dc = f3(m.a.x, m.a.y, m.a.z);
  const float n1_over_n2 = 1.0f / m.a.w;
  const float r_10 = m.b.x;
  const float a_x = m.b.y, a_y = m.b.z;
  const uint32_t dist = m.dist;
  const bool ms = m.model == MULTISCATTERING;
  const float z1 = rnd_tea(t);
  const float z2 = rnd_tea(t);
  const float3 mn = sample_visible_normal(dist, w_i, ffnormal, a_x, a_y, z1, z2, &capped);
  const float R_i = fresnel_interface(dot(w_i, mn), n1_over_n2);
  const float T_01_i = 1.0f - R_i;
  const float4 t4 = w.thr[pid];
  // direct illumination (:100-178)
  uint32_t li = (uint32_t)((float)S.n_lights * rnd_tea(t));
  if (li >= (uint32_t)S.n_lights) { li = (uint32_t)S.n_lights - 1; ++clamped; }
  const float light_pdf = 1.0f / (float)S.n_lights;
  const LightRaw ls = S.lights[li];
  float3 w_l, radiance;
  float ldist;
  eval_direct(S, hit_pos, ls, w_l, radiance, ldist, t, clamped);
  radiance = radiance / light_pdf;
  const float cos_theta_l = dot(ffnormal, w_l);
  if (cos_theta_l > 0.0f && !occluded(S, hit_pos, w_l, S.integ.scene_epsilon, ldist)) {
    const float3 Li = radiance;  // V * radiance with V = 1
    float3 add;
    if (ms) {  // :126-139
      const float3 lwi = to_local(w_i, ffnormal), lwl = to_local(w_l, ffnormal);
      add = Li * ms_diffuse_eval(dist, lwi, lwl, a_x, a_y, t, dc, 0u, &capped);
      add = add + Li * ms_conductor_eval(dist, lwi, lwl, m.eta, m.inv_eta, a_x, a_y, t, 0u, &capped);
    } else {  // :140-176
      const float3 refl_normal = normalize(w_i + w_l);
      const float R_refl = fresnel_interface(dot(refl_normal, w_l), n1_over_n2);
      const float T_01_diff = 1.0f - fresnel_interface(dot(mn, w_l), n1_over_n2);
      const float G_i_m_refl = masking_G1_aniso(dist, w_i, refl_normal, ffnormal, a_x, a_y);
      const float G_o_m_refl = masking_G1_aniso(dist, w_l, refl_normal, ffnormal, a_x, a_y);
      const float G_o_m_diff = masking_G1_aniso(dist, w_l, mn, ffnormal, a_x, a_y);
      const float D_refl = eval_visible_normal(dist, w_i, refl_normal, ffnormal, a_x, a_y);
      const float weight_refl = G_i_m_refl * G_o_m_refl * D_refl / (4.0f * fabsf(dot(w_i, ffnormal) * dot(w_l, ffnormal)));
      add = Li * kInvPi * cos_theta_l * dc * n1_over_n2 * n1_over_n2 * T_01_i * T_01_diff / (1.0f - dc * r_10) * G_o_m_diff;
      add = add + Li * R_refl * weight_refl;
    }
    emit = false;
    const float4 r = w.rad[pid];
    w.rad[pid] = make_float4(r.x + t4.x * add.x, r.y + t4.y * add.y, r.z + t4.z * add.z, 0.0f);
  }
  // indirect illumination (:181-289)
  const float xi = rnd_tea(t);
  float3 nd, weight;
  if (xi > R_i) {
    if (ms) {  // :187-218
      uint32_t order = 0;
      float3 wgt, lwm;
      nd = to_world(ms_diffuse_sample(dist, to_local(w_i, ffnormal), a_x, a_y, t, order, wgt, dc, lwm, &capped), ffnormal);
      const float T_01_r = 1.0f - fresnel_interface(dot(nd, to_world(lwm, ffnormal)), n1_over_n2);
      weight = f3s(n1_over_n2 * n1_over_n2 * T_01_r) / (1.0f - dc * r_10) * wgt;
    } else {  // :219-248
      nd = sample_cosine_weighted(mn, t);
      const float cos_theta_r = dot(nd, mn);
      const float G_o_m = masking_G1_aniso(dist, nd, mn, ffnormal, a_x, a_y);
      if (G_o_m < 0.0f) return false;
      const float T_01_r = 1.0f - fresnel_interface(cos_theta_r, n1_over_n2);
      weight = dc * n1_over_n2 * n1_over_n2 * T_01_r / (1.0f - dc * r_10) * G_o_m;
    }
  } else {
    if (ms) {  // :252-269 (the walk's Fresnel weight is not applied)
      uint32_t order = 10;
      float3 wgt;
      nd = to_world(ms_conductor_sample(dist, to_local(w_i, normal), m.eta, m.inv_eta, a_x, a_y, t, order, wgt, &capped), normal);
      weight = f3s(1.0f);
    } else {  // :270-287
      nd = reflect(d, mn);
      const float G_o_m = masking_G1_aniso(dist, nd, mn, ffnormal, a_x, a_y);
      if (G_o_m < 0.0f) return false;
      weight = f3s(G_o_m);
    }
  }
  const float3 nt = ld3(t4) * weight;
  w.ray_o[pid] = make_float4(hit_pos.x, hit_pos.y, hit_pos.z, 0.0f);
  w.ray_d[pid] = make_float4(nd.x, nd.y, nd.z, 0.0f);
  w.thr[pid] = make_float4(nt.x, nt.y, nt.z, 0.0f);
  return true;
}

// Layered materials: a Lambertian base under a dielectric interface.
//  * lambertian_interface_shader.cu:51-173 (smooth interface): the light sample's estimate carries the
//    interface's Fresnel transmittance in (T_01_i) and out (T_01_l) and the base's internal reflection
//    1 / (1 - rho r_10); its shadow ray (over [scene_epsilon, dist]) goes to the shadow queue.  With
//    probability 1 - R_i the path enters the base (cosine-weighted about the shading normal, weight
//    rho n^2 T_01_r / (1 - rho r_10)), otherwise it is mirrored about the shading normal with emission on.
//  * rough_diffuse_shader.cu:55-292 (rough interface): rough_diffuse_vertex, shadow ray inline.
// Neither is differentiable (pt_render_adjoint rejects them); the adjoint variant only settles the
// pending gradient of the previous vertex and replays the path.
template <bool kAdj>
__device__ __forceinline__ bool layered_path(const SceneDev& S, const WfDev& w, uint32_t pid, NeeRay& nee, bool& shadow, uint32_t& clamped, uint32_t& overflow, uint32_t& capped_total)
{
  bool cont = false;
  if constexpr (kAdj) apply_pending(S, w, pid);
  nee.eps = S.integ.scene_epsilon;
  const uint4 rg = w.rng[pid];
  const float4 h = w.hit[pid], o = w.ray_o[pid], d4 = w.ray_d[pid], t4 = w.thr[pid];
  const int depth = (int)(rg.w & META_DEPTH);
  if (depth <= S.integ.max_depth) {  // both shaders end the path at depth > max_depth
    const int prim = __float_as_int(h.w);
    const int4 info = __ldg(S.tri_info + prim);
    const MatDev& m = S.mats[info.w];
    const float3 d = ld3(d4);
    nee.o = ld3(o) + h.x * d;
    const float3 normal = shading_normal(S, info, h.y, h.z, prim);
    const float3 ffnormal = faceforward(normal, -d, normal);
    uint32_t t = rg.x;
    bool emit = (rg.w & META_EMIT) != 0;
    if (m.type == MAT_ROUGH_DIFFUSE) {
      int capped = 0;
      cont = rough_diffuse_vertex(S, w, pid, nee.o, d, normal, ffnormal, m, t, emit, clamped, capped);
      capped_total += capped;
    } else {
      const float3 dc = f3(m.a.x, m.a.y, m.a.z);
      const float n1_over_n2 = 1.0f / m.a.w, r_10 = m.b.x;
      const float R_i = fresnel_interface(dot(-d, ffnormal), n1_over_n2);
      const float T_01_i = 1.0f - R_i;
      const float draw = rnd_tea(t);
      uint32_t li = (uint32_t)((float)S.n_lights * draw);
      if (li >= (uint32_t)S.n_lights) { li = (uint32_t)S.n_lights - 1; ++clamped; }
      const float light_pdf = 1.0f / (float)S.n_lights;
      const LightRaw ls = S.lights[li];
      float3 radiance;
      float dist;
      eval_direct(S, nee.o, ls, nee.d, radiance, dist, t, clamped);
      radiance = radiance / light_pdf;
      const float cos_theta_l = dot(ffnormal, nee.d);
      if (cos_theta_l > 0.0f) {  // :95-118
        const float T_01_l = 1.0f - fresnel_interface(cos_theta_l, n1_over_n2);
        shadow = true;
        nee.tmax = dist;
        nee.c = ld3(t4) * (radiance * kInvPi * cos_theta_l * dc * n1_over_n2 * n1_over_n2 * T_01_l * T_01_i / (1.0f - dc * r_10));
        emit = false;
      }
      const float xi = rnd_tea(t);
      float3 nd, wgt;
      if (xi > R_i) {  // :127-153
        nd = sample_cosine_weighted(ffnormal, t);
        const float T_01_r = 1.0f - fresnel_interface(dot(nd, ffnormal), n1_over_n2);
        wgt = dc * n1_over_n2 * n1_over_n2 * T_01_r / (1.0f - dc * r_10);
      } else {  // :154-170
        nd = reflect(d, normal);
        wgt = f3s(1.0f);
        emit = true;
      }
      const float3 nt = ld3(t4) * wgt;
      w.ray_o[pid] = make_float4(nee.o.x, nee.o.y, nee.o.z, 0.0f);
      w.ray_d[pid] = make_float4(nd.x, nd.y, nd.z, 0.0f);
      w.thr[pid] = make_float4(nt.x, nt.y, nt.z, 0.0f);
      cont = true;
    }
    const uint32_t meta = push_md5_reset(w, pid, rg.w & META_KEEP, rg.y, rg.z, overflow);
    w.rng[pid] = make_uint4(t, rg.y, rg.z, meta | (uint32_t)(depth + 1) | (emit ? META_EMIT : 0u));
  }
  return cont;
}

// diffuse_shader.cu:42-107.  Adjoint: an albedo texel's gradient through the next-event estimate
// (resolved with the shadow ray) and through the bounce weight albedo / p (pending).
template <bool kAdj>
__device__ __forceinline__ bool diffuse_path(const SceneDev& S, const WfDev& w, uint32_t pid, NeeRay& nee, bool& shadow, uint32_t& clamped, uint32_t& overflow)
{
  bool cont = false;
  if constexpr (kAdj) apply_pending(S, w, pid);
  nee.eps = S.integ.scene_epsilon;
  // the path's records are loaded before the depth test (every queued id has them), so that their
  // latency overlaps the scene lookup
  uint4 rg = w.rng[pid];
  float4 h = w.hit[pid], o = w.ray_o[pid], d4 = w.ray_d[pid], t4 = w.thr[pid];
  int depth = (int)(rg.w & META_DEPTH);
  if (depth <= S.integ.max_depth) {
    int prim = __float_as_int(h.w);
    int4 info = __ldg(S.tri_info + prim);
    const MatDev& m = S.mats[info.w];
    float3 d = ld3(d4);
    nee.o = ld3(o) + h.x * d;
    float3 dc = f3(m.a.x, m.a.y, m.a.z);
    const int tid = __float_as_int(m.tmap.w);
    if (tid >= 0) {  // albedo texture (nearest texel of the cube map)
      const TexDev& T = S.tex[tid];
      const uint32_t tx = cube_texel(nee.o, ld3(m.tmap), T.w, T.h);
      dc = f3(__ldg(T.data + 3 * tx), __ldg(T.data + 3 * tx + 1), __ldg(T.data + 3 * tx + 2));
      nee.texel = ((uint32_t)tid << 24) | tx;
    }
    float3 normal = shading_normal(S, info, h.y, h.z, prim);
    float3 ffnormal = faceforward(normal, -d, normal);
    uint32_t t = rg.x;
    bool emit = (rg.w & META_EMIT) != 0;
    // uniform light pick and next-event estimation (:55-81)
    float draw = rnd_tea(t);
    if (S.n_lights > 0) {
      uint32_t li = (uint32_t)((float)S.n_lights * draw);
      if (li >= (uint32_t)S.n_lights) { li = (uint32_t)S.n_lights - 1; ++clamped; }
      float light_pdf = 1.0f / (float)S.n_lights;
      LightRaw ls = S.lights[li];
      float3 radiance;
      float dist;
      eval_direct(S, nee.o, ls, nee.d, radiance, dist, t, clamped);
      radiance = radiance / light_pdf;
      float cos_theta = dot(ffnormal, nee.d);
      if (cos_theta > 0.0f) {
        shadow = true;
        nee.tmax = dist - nee.eps;
        nee.c = ld3(t4) * (radiance * kInvPi * cos_theta * dc);
        emit = false;
      }
    }
    // Russian roulette on the mean albedo (:85-104)
    float prob = (dc.x + dc.y + dc.z) / 3.0f;
    float xi = rnd_tea(t);
    if (depth < S.integ.rr_start) prob = 1.0f;
    if (xi < prob || depth < S.integ.rr_start) {
      float3 nd = sample_cosine_weighted(ffnormal, t);
      float3 nt = ld3(t4) * (dc / prob);
      w.ray_o[pid] = make_float4(nee.o.x, nee.o.y, nee.o.z, 0.0f);
      w.ray_d[pid] = make_float4(nd.x, nd.y, nd.z, 0.0f);
      w.thr[pid] = make_float4(nt.x, nt.y, nt.z, 0.0f);
      cont = true;
      // weight albedo / p with p detached: d w / w = 1 / albedo per channel
      if (kAdj && nee.texel != kNoTexel)
        set_pending(w, pid, PEND_ALBEDO, (uint32_t)tid, nee.texel & 0xffffffu, f3(1.0f / dc.x, 1.0f / dc.y, 1.0f / dc.z));
    }
    const uint32_t meta = push_md5_reset(w, pid, rg.w & META_KEEP, rg.y, rg.z, overflow);
    w.rng[pid] = make_uint4(t, rg.y, rg.z, meta | (uint32_t)(depth + 1) | (emit ? META_EMIT : 0u));
  }
  return cont;
}

// metallic_shader.cu:45-161.  Adjoint: a GGX roughness texel's gradient through the weight, with
// the microfacet normal's sampling detached: d ln w / d alpha = d ln D(m) + d ln G1(wi) + d ln G1(wo)
// for the Walter and the visible-normal models alike.
// kMS: some conductor of the pass uses the multiple-scattering model (else that code is left out,
// which keeps the kernel's instruction footprint small).
template <bool kAdj, bool kMS>
__device__ __forceinline__ bool metal_path(const SceneDev& S, const WfDev& w, uint32_t pid, uint32_t& capped_total, uint32_t& overflow)
{
  bool cont = false;
  if constexpr (kAdj) apply_pending(S, w, pid);
  uint4 rg = w.rng[pid];
  float4 h = w.hit[pid], o = w.ray_o[pid], d4 = w.ray_d[pid];
  int depth = (int)(rg.w & META_DEPTH);
  if (depth < S.integ.max_depth) {
    int prim = __float_as_int(h.w);
    int4 info = __ldg(S.tri_info + prim);
    const MatDev& m = S.mats[info.w];
    float3 d = ld3(d4);
    float3 hit_point = ld3(o) + h.x * d;
    uint32_t rtexel = kNoTexel;
    float3 mn_used = f3s(0.0f);
    float3 normal = shading_normal(S, info, h.y, h.z, prim);
    float3 ffnormal = faceforward(normal, -d, normal);
    float3 w_i = -d;
    uint32_t seed = rg.x;
    float a_x = m.a.x, a_y = m.a.y;
    const int tid = __float_as_int(m.tmap.w);
    if (tid >= 0) {  // isotropic roughness texture (nearest texel of the cube map)
      const TexDev& T = S.tex[tid];
      rtexel = cube_texel(hit_point, ld3(m.tmap), T.w, T.h);
      a_x = a_y = __ldg(T.data + rtexel);
    }
    int capped = 0;
    float3 w_o, weight;
    bool go = true;
    if (kMS && m.model == MULTISCATTERING) {
      uint32_t order = 0;
      float3 lwo = ms_conductor_sample(m.dist, to_local(w_i, normal), m.eta, m.inv_eta, a_x, a_y, seed, order, weight, &capped);
      w_o = to_world(lwo, normal);
    } else {
      float z1 = rnd_tea(seed), z2 = rnd_tea(seed);
      float3 mn;
      float G_i_m, G_o_m;
      if (m.model == WALTER) {
        mn = sample_normal(m.dist, ffnormal, z1, z2, a_x);
        G_i_m = masking_G1(m.dist, w_i, mn, ffnormal, a_x);
      } else {
        mn = sample_visible_normal(m.dist, w_i, ffnormal, a_x, a_y, z1, z2, &capped);
        G_i_m = masking_G1_aniso(m.dist, w_i, mn, ffnormal, a_x, a_y);
      }
      go = G_i_m > 0.0f;
      if (go) {
        float3 F = fresnel_complex(w_i, mn, m.eta);
        w_o = -w_i + 2.0f * mn * dot(w_i, mn);
        float abs_i_m = fabsf(dot(w_i, mn)), abs_i_n = fabsf(dot(w_i, ffnormal)), abs_n_m = fabsf(dot(normal, mn));
        G_o_m = (m.model == WALTER) ? masking_G1(m.dist, w_o, mn, ffnormal, a_x) : masking_G1_aniso(m.dist, w_o, mn, ffnormal, a_x, a_y);
        go = G_o_m > 0.0f;
        weight = (m.model == WALTER) ? F * (abs_i_m * G_i_m * G_o_m / (abs_i_n * abs_n_m)) : F * G_o_m;
        mn_used = mn;
      }
    }
    capped_total += capped;
    if (go) {
      float4 t4 = w.thr[pid];
      float3 nt = ld3(t4) * weight;
      w.ray_o[pid] = make_float4(hit_point.x, hit_point.y, hit_point.z, 0.0f);
      w.ray_d[pid] = make_float4(w_o.x, w_o.y, w_o.z, 0.0f);
      w.thr[pid] = make_float4(nt.x, nt.y, nt.z, 0.0f);
      cont = true;
      if (kAdj && rtexel != kNoTexel && m.model != MULTISCATTERING && m.dist == GGX) {
        const float dl = ggx_dlnD(mn_used, ffnormal, a_x) + ggx_dlnG1(w_i, ffnormal, a_x) + ggx_dlnG1(w_o, ffnormal, a_x);
        set_pending(w, pid, PEND_ROUGH, (uint32_t)tid, rtexel, f3s(dl));
      }
    }
    const uint32_t meta = push_md5_reset(w, pid, rg.w & META_KEEP, rg.y, rg.z, overflow);
    w.rng[pid] = make_uint4(seed, rg.y, rg.z, meta | (uint32_t)(depth + 1) | META_EMIT);
  }
  return cont;
}

struct DirSeed {
  float3 dir;
  uint32_t seed;
};
// transparent_shader.cu:90-108: Fresnel reflectance about the shading normal (flipped, with the
// relative index inverted, when the ray is inside), one tea draw choosing the mirror or the refracted
// direction.
__device__ __forceinline__ DirSeed smooth_glass_dir(float3 d, float3 normal, float ior, float cos_theta, uint32_t t)
{
  const bool inside = cos_theta < 0.0f;
  const float n1_over_n2 = inside ? ior : 1.0f / ior;
  const float3 nn = inside ? -normal : normal;
  const float ci = inside ? -cos_theta : cos_theta;
  float R = 1.0f, ctt = 0.0f;
  const float st2 = n1_over_n2 * n1_over_n2 * (1.0f - ci * ci);
  if (st2 < 1.0f) {
    ctt = sqrtf(1.0f - st2);
    R = fresnel_R(ci, ctt, n1_over_n2);
  }
  const float reflect_xi = rnd_tea(t);
  DirSeed r;
  r.dir = reflect_xi < R ? reflect(d, nn) : n1_over_n2 * d + nn * (n1_over_n2 * ci - ctt);
  r.seed = t;
  return r;
}

// rough_transparent_shader.cu:66-225, and transparent_shader.cu:47-115 for smooth glass (Beer roulette
// inside, then the Fresnel choice between the mirror and the refracted direction about the shading
// normal).  No parameters to differentiate: the adjoint only settles the pending gradient of the
// previous vertex.
// kMS: some rough dielectric of the pass uses the multiple-scattering model (as for k_shade_metal).
template <bool kAdj, bool kMS>
__device__ __forceinline__ bool glass_path(const SceneDev& S, const WfDev& w, uint32_t pid, uint32_t& capped_total, uint32_t& overflow)
{
  bool cont = false;
  if constexpr (kAdj) apply_pending(S, w, pid);
  uint4 rg = w.rng[pid];
  float4 h = w.hit[pid], o = w.ray_o[pid], d4 = w.ray_d[pid];
  int depth = (int)(rg.w & META_DEPTH);
  // rough_transparent_shader.cu:68 ends paths at depth >= max_depth, transparent_shader.cu:50 at depth > max_depth
  if (depth < S.integ.max_depth ||
      (depth == S.integ.max_depth && S.mats[__ldg(&S.tri_info[__float_as_int(h.w)].w)].type == MAT_TRANSPARENT)) {
    int prim = __float_as_int(h.w);
    int4 info = __ldg(S.tri_info + prim);
    const MatDev& m = S.mats[info.w];
    const bool smooth = m.type == MAT_TRANSPARENT;
    const float ior = m.a.x, rough = m.a.y;
    float3 d = ld3(d4);
    float3 hit_point = ld3(o) + h.x * d;
    float3 normal = shading_normal(S, info, h.y, h.z, prim);
    float3 ffnormal = faceforward(normal, -d, normal);
    float3 w_i = -d;
    uint32_t t = rg.x;
    float3 beam_T = f3s(1.0f);
    bool go = true;
    float cos_theta = dot(-d, normal);
    if (cos_theta < 0.0f) {  // Beer absorption with Russian roulette inside (:84-91)
      beam_T = expf3((-h.x) * f3(m.b.x, m.b.y, m.b.z));
      float prob = (beam_T.x + beam_T.y + beam_T.z) / 3.0f;
      if (rnd_tea(t) >= prob) go = false;
      else beam_T = beam_T / prob;
    }
    int capped = 0;
    float3 w_o;
    float3 weight = f3s(1.0f);
    if (go && smooth) {
      const DirSeed ds = smooth_glass_dir(d, normal, ior, cos_theta, t);
      w_o = ds.dir;
      t = ds.seed;
    } else if (go) {
      float z1 = rnd_tea(t), z2 = rnd_tea(t);
      if (kMS && m.model == MULTISCATTERING) {  // :100-120
        uint32_t order = 0;
        float3 lwo = ms_dielectric_sample(m.dist, to_local(w_i, normal), 1.0f / ior, rough, rough, t, order, &capped);
        w_o = to_world(lwo, normal);
      } else {
        float3 mn = (m.model == WALTER) ? sample_normal(m.dist, ffnormal, z1, z2, rough)
                                        : sample_visible_normal(m.dist, w_i, ffnormal, rough, rough, z1, z2, &capped);
        float cos_in = dot(normal, w_i);
        float eta = cos_in < 0.0f ? ior : 1.0f / ior;
        float G_i_m = (m.model == WALTER) ? masking_G1(m.dist, w_i, mn, ffnormal, rough) : masking_G1_aniso(m.dist, w_i, mn, ffnormal, rough, rough);
        go = G_i_m > 0.0f;
        if (go) {
          // get_rough_glass_rays (:39-55)
          float ct = fabsf(dot(mn, -d));
          float st2 = eta * eta * (1.0f - ct * ct);
          float ctt = sqrtf(1.0f - st2);
          float R = st2 < 1.0f ? fresnel_R(ct, ctt, eta) : 1.0f;
          float3 refr = eta * d + mn * (eta * ct - ctt);
          float3 refl = reflect(d, mn);
          float abs_i_m = fabsf(dot(w_i, mn)), abs_i_n = fabsf(dot(w_i, ffnormal)), abs_n_m = fabsf(dot(normal, mn));
          float rr = rnd_tea(t);
          w_o = rr > R ? refr : refl;
          float G_o_m = (m.model == WALTER) ? masking_G1(m.dist, w_o, mn, ffnormal, rough) : masking_G1_aniso(m.dist, w_o, mn, ffnormal, rough, rough);
          go = G_o_m > 0.0f;
          float wgt = (m.model == WALTER) ? abs_i_m * G_i_m * G_o_m / (abs_i_n * abs_n_m) : G_o_m;
          weight = f3s(wgt);
        }
      }
    }
    capped_total += capped;
    if (go) {
      float4 t4 = w.thr[pid];
      float3 nt = ld3(t4) * weight * beam_T;
      w.ray_o[pid] = make_float4(hit_point.x, hit_point.y, hit_point.z, 0.0f);
      w.ray_d[pid] = make_float4(w_o.x, w_o.y, w_o.z, 0.0f);
      w.thr[pid] = make_float4(nt.x, nt.y, nt.z, 0.0f);
      cont = true;
    }
    const uint32_t meta = smooth ? (rg.w & META_KEEP) : push_md5_reset(w, pid, rg.w & META_KEEP, rg.y, rg.z, overflow);
    w.rng[pid] = make_uint4(t, rg.y, rg.z, meta | (uint32_t)(depth + 1) | META_EMIT);
  }
  return cont;
}

// ------------------------------------------------------------------ translucent objects
// rough_subsurface_scattering_shader.cu:56-455 (REFLECT, TRANSMIT, DIRECTLIGHT and RND_64 defined),
// one vertex: the microfacet normal from two MD5 draws; a light picked with an MD5 draw and its
// reflection-only estimate (the multiscatter model: the multiscatter dielectric BSDF), with the shadow
// ray traced here because the multiscatter evaluation draws tea randoms only when the light is
// visible; then the smooth shader's Beer roulette and Fresnel choice on the microfacet normal, the
// refraction / reflection weight on the child, and on a refraction from outside the dipole gather
// (pushed with that weight; its draws must also exceed 0.001).  Returns whether the path continues.
static __device__ bool rough_translucent_vertex(const SceneDev& S, const WfDev& w, uint32_t pid, const uint4& rg, int depth, const float4& h,
                                         const float4& o, const float4& d4, const int4& info, const MatDev& m, const ScatDev& P,
                                         uint32_t& overflow, uint32_t& clamped, int& capped)
{
  const float3 d = ld3(d4);
  float3 normal = shading_normal(S, info, h.y, h.z, __float_as_int(h.w));
  const float3 ffnormal = faceforward(normal, -d, normal);
  const float3 hit_pos = ld3(o) + h.x * d;
  const float3 w_i = -d;
  float recip_ior = 1.0f / P.relative_ior;
  float3 beam_T = f3s(1.0f);
  uint32_t t = rg.x;
  uint2 t64 = make_uint2(rg.y, rg.z);
  const float reflect_xi = rnd_md5(t64);
  const float z1 = rnd_md5(t64);
  const float z2 = rnd_md5(t64);
  const float a_x = m.a.y, a_y = m.a.z;
  const uint32_t model = __float_as_uint(m.a.w), dist = m.dist;
  const float3 mn = model == WALTER ? sample_normal(dist, ffnormal, z1, z2, a_x) : sample_visible_normal(dist, w_i, ffnormal, a_x, a_y, z1, z2, &capped);
  const float cos_theta_i = dot(w_i, mn);
  const bool inside = dot(w_i, normal) < 0.0f;
  bool emit = (rg.w & META_EMIT) != 0;
  const float4 t4 = w.thr[pid];
  // light sample (:93-152)
  uint32_t li = (uint32_t)((float)S.n_lights * rnd_md5(t64));
  if (li >= (uint32_t)S.n_lights) { li = (uint32_t)S.n_lights - 1; ++clamped; }
  const float light_pdf = 1.0f / (float)S.n_lights;
  const LightRaw ls = S.lights[li];
  float3 w_l, light_radiance;
  float ldist;
  eval_direct(S, hit_pos, ls, w_l, light_radiance, ldist, t, clamped);
  light_radiance = light_radiance / light_pdf;
  const float cos_l = dot(ffnormal, w_l);
  if (!inside && cos_l > 0.0f) {
    const float V = occluded(S, hit_pos, w_l, S.integ.scene_epsilon, ldist) ? 0.0f : 1.0f;
    if (V > 0.0f) {
      const float3 Li = V * light_radiance;
      float3 add;
      if (model == MULTISCATTERING) {
        const float brdf = ms_dielectric_eval(dist, to_local(w_i, ffnormal), to_local(w_l, ffnormal), recip_ior, a_x, a_y, t, 0u, &capped);
        add = Li * brdf;
        emit = false;
      } else {
        const float3 rn = normalize(w_i + w_l);
        const float cr = dot(rn, w_l);
        float Rr = 1.0f;
        const float st2 = recip_ior * recip_ior * (1.0f - cr * cr);
        if (st2 < 1.0f) Rr = fresnel_R(cr, sqrtf(1.0f - st2), recip_ior);
        const float Gi = masking_G1_aniso(dist, w_i, rn, ffnormal, a_x, a_y);
        const float Go = masking_G1_aniso(dist, w_l, rn, ffnormal, a_x, a_y);
        const float D = eval_visible_normal(dist, w_i, rn, ffnormal, a_x, a_y);
        const float wr = Gi * Go * D / (4.0f * fabsf(dot(w_i, ffnormal) * dot(w_l, ffnormal)));
        add = Li * Rr * wr;
        emit = true;
      }
      const float4 r = w.rad[pid];
      w.rad[pid] = make_float4(r.x + t4.x * add.x, r.y + t4.y * add.y, r.z + t4.z * add.z, 0.0f);
    }
  }
  uint32_t meta = rg.w & META_KEEP;
  bool cont = false, gather = false, child_emit = true;
  float3 nd = f3s(0.0f), weight = f3s(1.0f);
  auto roulette_inside = [&]() -> bool {  // Beer transmittance inside, as the smooth shader
    const float3 ext = m.model == DIRECTIONAL_DIPOLE ? P.deltaEddExtinction : P.extinction;
    beam_T = expf3((-h.x) * ext);
    const float prob = (beam_T.x + beam_T.y + beam_T.z) / 3.0f;
    if (rnd_md5(t64) >= prob) return false;
    beam_T = beam_T / prob;
    recip_ior = P.relative_ior;
    normal = -normal;
    return true;
  };
  if (model == WALTER || model == VISIBLE_NORMALS) {
    if (!inside || roulette_inside()) {
      const float st2 = recip_ior * recip_ior * (1.0f - cos_theta_i * cos_theta_i);
      float cos_t = 1.0f, R = 1.0f;
      if (st2 < 1.0f) {
        cos_t = sqrtf(1.0f - st2);
        R = fresnel_R(cos_theta_i, cos_t, recip_ior);
      }
      if (reflect_xi >= R) {
        nd = recip_ior * (cos_theta_i * mn - w_i) - mn * cos_t;
        gather = !inside;
      } else {
        nd = 2.0f * cos_theta_i * mn - w_i;
        child_emit = emit;
      }
      if (model == WALTER) {
        const float G_i_m = masking_G1(dist, w_i, mn, ffnormal, a_x);
        const float abs_i_m = fabsf(dot(w_i, mn)), abs_i_n = fabsf(dot(w_i, ffnormal)), abs_n_m = fabsf(dot(ffnormal, mn));
        const float G_o_m = masking_G1(dist, nd, mn, ffnormal, a_x);
        weight = f3s(1.0f) * (abs_i_m * G_i_m * G_o_m / (abs_i_n * abs_n_m));
      } else {
        weight = f3s(1.0f) * masking_G1_aniso(dist, nd, mn, ffnormal, a_x, a_y);
      }
      cont = true;
    }
  } else {  // MULTISCATTERING_MODEL (:287-452)
    uint32_t order = 0;
    const float3 w_o = to_world(ms_dielectric_sample(dist, to_local(w_i, normal), 1.0f / P.relative_ior, a_x, a_y, t, order, &capped), normal);
    const bool is_refraction = dot(w_o, ffnormal) < 0.0f;
    if (!inside || roulette_inside()) {
      nd = w_o;
      gather = is_refraction && !inside;
      cont = true;
    }
  }
  if (cont) {
    if (gather && !(rg.w & META_PROBE)) {
      const uint32_t slot = meta >> META_GSHIFT;
      if (slot < w.g_slots) {
        size_t at = (size_t)slot * w.cap + pid;
        w.g_a[at] = make_float4(hit_pos.x, hit_pos.y, hit_pos.z, t4.x);
        w.g_b[at] = make_float4(normal.x, normal.y, normal.z, t4.y);
        w.g_c[at] = make_float2(t4.z, __int_as_float(info.w));
        w.g_d[at] = make_float4(weight.x, weight.y, weight.z, 1.0f);
        meta += 1u << META_GSHIFT;
      } else {
        ++overflow;
      }
    }
    const float3 nt = ld3(t4) * weight * beam_T;
    w.ray_o[pid] = make_float4(hit_pos.x, hit_pos.y, hit_pos.z, 0.0f);
    w.ray_d[pid] = make_float4(nd.x, nd.y, nd.z, 0.0f);
    w.thr[pid] = make_float4(nt.x, nt.y, nt.z, 0.0f);
  }
  w.rng[pid] = make_uint4(t, t64.x, t64.y, meta | (uint32_t)(depth + 1) | (child_emit ? META_EMIT : 0u));
  return cont;
}

// subsurface_scattering_shader.cu:55-201 with REFLECT, TRANSMIT and RND_64 defined: the Fresnel
// choice between the reflected and the refracted ray (one MD5 draw), and inside the object Beer
// transmittance over the segment with Russian roulette on its mean (extinction, or the
// delta-Eddington extinction for the directional dipole).  A camera path refracted into the object
// from outside also owes the dipole gather over the frame's probes (:126-173).  The reference
// evaluates it after the refracted subtree has returned, so its MD5 draws follow every draw of that
// subtree; the vertex (position, normal, throughput, material) is therefore pushed on the path's
// gather stack and evaluated in last-in first-out order when the path has ended (k_gather).  A
// probe's indirect path does not gather: in the reference it would read the probe buffer that its
// own launch is writing.
//
// Adjoint: the gather a camera path owes at an entry vertex is taken off R there (its forward value
// was stored with the path); its gradient is added at the end (k_gather<true>).  Inside, the weight
// beam_T / p has p detached: d w / d sigma_a / w = -t * scale per channel.
template <bool kAdj, bool kRough>
__device__ __forceinline__ bool translucent_path(const SceneDev& S, const WfDev& w, uint32_t pid, uint32_t& overflow, uint32_t& clamped, int& capped)
{
  bool cont = false;
  if constexpr (kAdj) apply_pending(S, w, pid);
  uint4 rg = w.rng[pid];
  float4 h = w.hit[pid], o = w.ray_o[pid], d4 = w.ray_d[pid];
  int depth = (int)(rg.w & META_DEPTH);
  if (depth <= S.integ.max_depth) {
    int prim = __float_as_int(h.w);
    int4 info = __ldg(S.tri_info + prim);
    const MatDev& m = S.mats[info.w];
    const ScatDev& P = S.scat[info.w];
    if (kRough && m.type == MAT_ROUGH_TRANSLUCENT) {
      if constexpr (kRough) cont = rough_translucent_vertex(S, w, pid, rg, depth, h, o, d4, info, m, P, overflow, clamped, capped);
    } else {
    float3 d = ld3(d4);
    float3 no = shading_normal(S, info, h.y, h.z, prim);
    float3 xo = ld3(o) + h.x * d;
    float3 wo = -d;
    float recip_ior = 1.0f / P.relative_ior;
    float3 beam_T = f3s(1.0f);
    uint2 t64 = make_uint2(rg.y, rg.z);
    float reflect_xi = rnd_md5(t64);
    float cos_o = dot(wo, no);
    bool inside = cos_o < 0.0f;
    bool alive = true;
    if (inside) {
      float3 ext = m.model == DIRECTIONAL_DIPOLE ? P.deltaEddExtinction : P.extinction;
      beam_T = expf3((-h.x) * ext);
      float prob = (beam_T.x + beam_T.y + beam_T.z) / 3.0f;
      if (rnd_md5(t64) >= prob) {
        alive = false;
      } else {
        beam_T = beam_T / prob;
        recip_ior = P.relative_ior;
        no = -no;
        cos_o = -cos_o;
      }
    }
    uint32_t meta = rg.w & META_KEEP;
    if (alive) {
      float st2 = recip_ior * recip_ior * (1.0f - cos_o * cos_o);
      float cos_t = 1.0f, R = 1.0f;
      if (st2 < 1.0f) {
        cos_t = sqrtf(1.0f - st2);
        R = fresnel_R(cos_o, cos_t, recip_ior);
      }
      float4 t4 = w.thr[pid];
      float3 nd;
      if (reflect_xi >= R) {
        nd = recip_ior * (cos_o * no - wo) - no * cos_t;
        if (!inside && !(rg.w & META_PROBE)) {
          uint32_t slot = meta >> META_GSHIFT;
          if (slot < w.g_slots) {
            size_t at = (size_t)slot * w.cap + pid;
            w.g_a[at] = make_float4(xo.x, xo.y, xo.z, t4.x);
            w.g_b[at] = make_float4(no.x, no.y, no.z, t4.y);
            w.g_c[at] = make_float2(t4.z, __int_as_float(info.w));
            w.g_d[at] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
            if constexpr (kAdj) {
              const ItemDev& it = w.items[w.path_item[pid]];
              const uint64_t local = pid - it.path_begin;
              const uint64_t gp = (uint64_t)(it.first_frame + (uint32_t)(local / it.pixels) - S.adj_first) * it.pixels + local % it.pixels;
              const float4 G = S.adj_G[gp * S.adj_slots + slot];
              const float4 r = w.rad[pid];
              w.rad[pid] = make_float4(r.x - t4.x * G.x, r.y - t4.y * G.y, r.z - t4.z * G.z, 0.0f);
            }
            meta += 1u << META_GSHIFT;
          } else {
            ++overflow;
          }
        }
      } else {
        nd = 2.0f * cos_o * no - wo;
      }
      float3 nt = ld3(t4) * beam_T;
      w.ray_o[pid] = make_float4(xo.x, xo.y, xo.z, 0.0f);
      w.ray_d[pid] = make_float4(nd.x, nd.y, nd.z, 0.0f);
      w.thr[pid] = make_float4(nt.x, nt.y, nt.z, 0.0f);
      cont = true;
      if (kAdj && inside) set_pending(w, pid, PEND_SIGMA, (uint32_t)info.w, 0u, f3s(-h.x * m.a.x));
    }
    w.rng[pid] = make_uint4(rg.x, t64.x, t64.y, meta | (uint32_t)(depth + 1) | META_EMIT);
    }
  }
  return cont;
}

// ------------------------------------------------------------------ conductor and dielectric shading kernels
template <bool kAdj, bool kMS>
__global__ void __launch_bounds__(kBlock) k_shade_metal(WfDev w)
{
  __shared__ uint32_t sm[kWarps + 1];
  const uint32_t n = w.cnt[CNT_Q_METAL];
  const uint32_t* q = w.q_mat + (size_t)QC_METAL * w.cap;
  uint32_t capped_total = 0;
  uint32_t overflow = 0;
  for (uint32_t base = blockIdx.x * kBlock; base < n; base += gridDim.x * kBlock) {
    uint32_t i = base + threadIdx.x;
    bool cont = false;
    uint32_t pid = 0;
    if (i < n) {
      pid = q[i];
      cont = metal_path<kAdj, kMS>(scene_of(w, pid), w, pid, capped_total, overflow);
    }
    uint32_t c_slot = block_slot(cont, w.cnt + w.out_slot, sm);
    if (cont) w.q_out[c_slot] = pid;
  }
  if (capped_total) atomicAdd(cnt64(w.cnt, CNT_CAPPED), (unsigned long long)capped_total);
  if (overflow) atomicAdd(cnt64(w.cnt, CNT_ERROR), (unsigned long long)overflow);
}
template <bool kAdj, bool kMS>
__global__ void __launch_bounds__(kBlock) k_shade_glass(WfDev w)
{
  __shared__ uint32_t sm[kWarps + 1];
  const uint32_t n = w.cnt[CNT_Q_GLASS];
  const uint32_t* q = w.q_mat + (size_t)QC_GLASS * w.cap;
  uint32_t capped_total = 0;
  uint32_t overflow = 0;
  for (uint32_t base = blockIdx.x * kBlock; base < n; base += gridDim.x * kBlock) {
    uint32_t i = base + threadIdx.x;
    bool cont = false;
    uint32_t pid = 0;
    if (i < n) {
      pid = q[i];
      cont = glass_path<kAdj, kMS>(scene_of(w, pid), w, pid, capped_total, overflow);
    }
    uint32_t c_slot = block_slot(cont, w.cnt + w.out_slot, sm);
    if (cont) w.q_out[c_slot] = pid;
  }
  if (capped_total) atomicAdd(cnt64(w.cnt, CNT_CAPPED), (unsigned long long)capped_total);
  if (overflow) atomicAdd(cnt64(w.cnt, CNT_ERROR), (unsigned long long)overflow);
}

// One full wave of a grid-stride kernel: the SM count times the blocks of kBlock threads that fit on an
// SM at the kernel's register and shared-memory use (cached per kernel and thread).
template <class K> inline int full_wave(K kernel)
{
  static thread_local std::vector<std::pair<const void*, int>> cache;
  const void* key = reinterpret_cast<const void*>(kernel);
  for (const auto& e : cache)
    if (e.first == key) return e.second;
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, kBlock, 0) != cudaSuccess || blocks < 1) blocks = 8;
  const int grid = sm_count() * blocks;
  cache.emplace_back(key, grid);
  return grid;
}

// ------------------------------------------------------------------ path pools and large vertex programs (pt_pool.cu, pt_pool_all.cu)
// All bounces of the paths in the queue w.q_in (at most n of them) by path pools.  `programs`: the vertex
// programs the pass needs beside diffuse, conductor, dielectric, emitter and miss.
// Up to how many paths a chunk runs through pools instead of the wavefront's launches.  A bounce of the
// wavefront costs eleven launches and waits for its slowest ray on the whole GPU, which a small chunk
// cannot hide; a pool's warps wait for their block's slowest ray instead, and its one kernel holds every
// program, which a large chunk pays for.  The other contexts' work fills the wavefront's gaps where several
// render at once, so the lines lie lower there, and that is where those of one scene are drawn: a program
// that renders in one context alone could go on to about twice the paths.  Measured (wavefront / pools, us a
// render; three contexts in turn, then one alone):
//   basic (subdiv 5, depth 8)   0.79 M paths 1888 / 1673, 2182 / 1816; 1.57 M 3023 / 3111, 3445 / 3247
//   layered, multiple scattering   0.52 M 2680 / 2656, 3769 / 2780; 1.05 M 3923 / 4011, 4998 / 4276
//   smooth translucent   1.57 M 3894 / 3263, 4713 / 3619; 2.1 M 4810 / 4236, 5583 / 4584
//   translucent and all programs   1.57 M 4423 / 4055, 5496 / 4431 (rough, Walter), 5509 / 5220, 6728 / 5718 (rough,
//   multiple scattering), 7922 / 7015, 10004 / 7563 (beside layered); 2.1 M 5414 / 5250, 6782 / 6771, 9813 / 9082
// Passes of several scenes (the wavefront's multi-scene traversal spills; four scenes in one batch):
//   basic   1.05 M 2881 / 2600, 2.1 M 4638 / 4805; layered   1.05 M 5225 / 4605, 4.2 M 14576 / 14887
//   smooth translucent   4.2 M 9672 / 9137, 8.4 M 17746 / 17688, 12.6 M 25939 / 26366
//   translucent and all programs   2.1 M 8276 / 7693 (one scene of each kind), 7977 / 7487 (rough), 11685 / 10055 (beside
//   layered); 4.2 M 12670 / 14277, 13586 / 13889, 19860 / 18731; 8.4 M 21870 / 27563
inline uint64_t pool_max_paths(bool translucent, bool all_programs, bool multi)
{
  if (multi && translucent) return all_programs ? 1ull << 21 : 1ull << 23;
  const uint64_t single = translucent ? 3ull << 19 : all_programs ? 1ull << 19 : 3ull << 18;
  return multi ? 2 * single : single;
}
enum PoolPrograms { POOL_BASIC = 0, POOL_TRANSLUCENT = 1 /* and smooth translucent objects */, POOL_ALL = 2 };
pt_status launch_path_pools(const SceneDev& S0, const WfDev& w, uint64_t n, bool multi, bool adjoint, PoolPrograms programs, int refill,
                            cudaStream_t stream);
pt_status launch_path_pools_all(const SceneDev& S0, const WfDev& w, uint64_t n, bool multi, bool adjoint, int refill, cudaStream_t stream);
// The wavefront's layered and translucent shading, and the conductors and dielectrics of a pass that holds
// the multiple-scattering model.
void launch_shade_layered(const WfDev& w, bool adjoint, cudaStream_t stream);
void launch_shade_translucent(const WfDev& w, bool adjoint, bool rough, cudaStream_t stream);
void launch_shade_ms(const WfDev& w, bool adjoint, cudaStream_t stream);

}  // namespace pt
