// Wavefront path tracer: the sm_100a replacement for the recursive OptiX launch of
// OptixScene::renderScene (OptixScene.cpp:159) running path_tracer.cu and the material programs.
//
// One call of pt_render_frames traces every (pixel, frame) camera sample of a group of frames at
// once.  Per bounce:
//   extend   closest hit through the BVH; the class of each ray's hit (miss, emitter, diffuse, conductor,
//            rough dielectric, translucent, layered) is recorded by queue position
//   bin      a stable partition of the queue by class into the material queues -- the sort by material
//            key -- (warp ballots + shared-memory prefix per block, a scan over the blocks)
//   shade    one kernel per material class, following diffuse_shader.cu, metallic_shader.cu,
//            rough_transparent_shader.cu, arealight_shader.cu, constantbg.cu; continuing paths are
//            appended to the next active queue and diffuse next-event estimation to the shadow queue
//   shadow   any-hit through the same BVH; unoccluded contributions are added to the path radiance
// (a chunk of few paths runs all of its bounces in one launch of path pools instead, pt_pool.cuh)
// and finally `accumulate` folds the frames into the float4 running mean in frame order
// (path_tracer.cu:64-68).
//
// Scenes with translucent objects first run the probe pass of every frame (sample_camera.cu): one
// PositionSample per (object, sample), lit by a shadowed light sample or by an indirect path that
// goes through the same wavefront.  The probes with L != 0 are compacted in order, and the dipole
// gathers that camera paths owe on entering a translucent object are evaluated after the paths end
// (see k_shade_translucent).  Each path keeps one tea stream and one MD5 stream exactly as the
// reference's recursion passes prd.seed down the path, so paths consume identical random numbers.
//
// The reference's recursion result is result = own + child * weight; here the equivalent iterative
// form is used: radiance += throughput * own, throughput *= weight.
//
// All queue counts live in device memory and every kernel reads its count there, so a whole render
// is a fixed sequence of launches with no host synchronisation (CUDA-graph capturable).
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "pt_context.h"
#include "pt_dipole.cuh"
#include "pt_wavefront.cuh"

namespace pt {

// Threads per block of the persistent traversal kernels, and the resident blocks per SM they are
// compiled for (register budget: 1,024 threads per SM at 64 registers).
#ifndef PT_TRACE_BLOCK
#define PT_TRACE_BLOCK 128
#endif
#ifndef PT_TRACE_MIN_BLOCKS
#define PT_TRACE_MIN_BLOCKS (1024 / PT_TRACE_BLOCK)
#endif
constexpr int kTraceBlock = PT_TRACE_BLOCK;
// A value with its derivatives with respect to (sigma_a, sigma_s') of one channel.
struct Dual2 {
  float v, da, ds;
};
// The standard dipole of one channel (standard_dipole.h:8-29) and its derivatives with respect to the
// channel's sigma_a and sigma_s' (before the material's scale; A depends on the ior only):
// ln S_r = ln 3D + ln(1 + tr d_r) - tr d_r - 3 ln d_r, and likewise for the virtual source.
__device__ __forceinline__ Dual2 dipole_channel_grad(float dist, float sa, float red_ext, float A, float scale)
{
  const float x = red_ext;             // sigma_t' (scaled)
  const float D = 1.0f / (3.0f * x);
  const float dD = -D / x * scale;     // d D / d sigma (either), sigma_t' = (sigma_s' + sigma_a) * scale
  const float three_D = 3.0f * D, d3D = 3.0f * dD;
  const float tr = sqrtf(sa / D);      // sqrt(3 sigma_a sigma_t')
  const float dtr_a = 3.0f * scale * (x + sa) / (2.0f * tr), dtr_s = 3.0f * sa * scale / (2.0f * tr);
  const float ext = 4.0f * A * D, dext = 4.0f * A * dD;
  const float r2 = dist * dist;
  const float dr2 = r2 + three_D * three_D, dr = sqrtf(dr2), ddr = three_D * d3D / dr;
  const float dv2 = r2 + ext * ext, dv = sqrtf(dv2), ddv = ext * dext / dv;
  const float cmf = three_D + ext, dcmf = d3D + dext;
  const float trr = tr * dr, trv = tr * dv;
  const float Sr = three_D * (1.0f + trr) / (dr2 * dr) * expf(-trr);
  const float Sv = cmf * (1.0f + trv) / (dv2 * dv) * expf(-trv);
  // d(tr d) for each of the two parameters
  const float dtrr_a = dtr_a * dr + tr * ddr, dtrr_s = dtr_s * dr + tr * ddr;
  const float dtrv_a = dtr_a * dv + tr * ddv, dtrv_s = dtr_s * dv + tr * ddv;
  const float kr_a = d3D / three_D + dtrr_a / (1.0f + trr) - dtrr_a - 3.0f * ddr / dr;
  const float kr_s = d3D / three_D + dtrr_s / (1.0f + trr) - dtrr_s - 3.0f * ddr / dr;
  const float kv_a = dcmf / cmf + dtrv_a / (1.0f + trv) - dtrv_a - 3.0f * ddv / dv;
  const float kv_s = dcmf / cmf + dtrv_s / (1.0f + trv) - dtrv_s - 3.0f * ddv / dv;
  return Dual2{Sr + Sv, Sr * kr_a + Sv * kv_a, Sr * kr_s + Sv * kv_s};
}

// ------------------------------------------------------------------ kernels
// path_tracer.cu:32-60: seed, jitter, pinhole direction; paths outside the patch are flagged.
// kAdj: the adjoint replay; the path's radiance slot carries R (the forward radiance of the path, not
// yet passed by the replay) and adj_a its image gradient.
template <bool kAdj>
__global__ void __launch_bounds__(kBlock) k_raygen(WfDev w, uint64_t n_paths)
{
  __shared__ uint32_t sm[kWarps + 1];
  for (uint64_t base = (uint64_t)blockIdx.x * kBlock; base < n_paths; base += (uint64_t)gridDim.x * kBlock) {
    uint64_t pid = base + threadIdx.x;
    bool valid = pid < n_paths;
    bool inside = false;
    if (valid) {
      uint32_t k = find_item(w.items, w.n_items, pid, [](const ItemDev& it) { return it.path_begin; });
      const ItemDev& it = w.items[k];
      const SceneDev& S = w.scenes[it.scene];
      const CameraDev& C = S.cam;
      w.path_item[pid] = (uint16_t)k;
      uint64_t local = pid - it.path_begin;
      uint32_t fl = (uint32_t)(local / it.pixels), p = (uint32_t)(local % it.pixels);
      uint32_t x = p % C.width, y = p / C.width;
      uint32_t frame = it.first_frame + fl;
      inside = !(x < C.patch_origin.x || x > C.patch_origin.x + C.patch_dims.x || y < C.patch_origin.y || y > C.patch_origin.y + C.patch_dims.y);
      if (inside) {
        uint32_t seed = tea16(C.width * y + x, frame);
        uint2 s64 = make_uint2(seed, seed);
        float jx = rnd_tea(seed);
        float jy = rnd_tea(seed);
        float ipx = ((float)x + jx) / (float)C.width * 2.0f - 1.0f;
        float ipy = ((float)y + jy) / (float)C.height * 2.0f - 1.0f;
        float3 dir = normalize(ipx * C.U + ipy * C.V + C.W);
        w.ray_o[pid] = make_float4(C.eye.x, C.eye.y, C.eye.z, 0.0f);
        w.ray_d[pid] = make_float4(dir.x, dir.y, dir.z, 0.0f);
        w.thr[pid] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
        if constexpr (kAdj) {
          const uint64_t gp = (uint64_t)(frame - S.adj_first) * it.pixels + p;
          const float4 L = S.adj_L[gp];
          const float4 di = S.adj_dimg[p];
          // the running mean skips non-finite samples (path_tracer.cu:64-68): no gradient through them
          const bool fin = isfinite(L.x) && isfinite(L.y) && isfinite(L.z);
          const float sc = fin ? S.adj_dscale : 0.0f;
          w.rad[pid] = make_float4(L.x, L.y, L.z, 0.0f);
          w.adj_a[pid] = make_float4(di.x * sc, di.y * sc, di.z * sc, __uint_as_float(PEND_NONE));
        } else {
          w.rad[pid] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        w.rng[pid] = make_uint4(seed, s64.x, s64.y, META_EMIT);
      } else {
        w.rad[pid] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        w.rng[pid] = make_uint4(0, 0, 0, META_OUTSIDE);
      }
    }
    uint32_t slot = block_slot(inside, w.cnt + w.in_slot, sm);
    if (inside) w.q_in[slot] = (uint32_t)pid;
  }
}

__global__ void __launch_bounds__(kBlock) k_extend(WfDev w)
{
  const uint32_t n = w.cnt[w.in_slot];
  uint32_t traced = 0;
  for (uint32_t base = blockIdx.x * kBlock; base < n; base += gridDim.x * kBlock) {
    uint32_t i = base + threadIdx.x;
    int cls = -1;
    uint32_t pid = 0;
    if (i < n) {
      pid = w.q_in[i];
      const SceneDev& S = scene_of(w, pid);
      float4 o = w.ray_o[pid], d = w.ray_d[pid];
      Hit h = scene_closest(S, ld3(o), ld3(d), S.integ.scene_epsilon, kDefaultMax);
      w.hit[pid] = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
      if (h.prim < 0) cls = QC_MISS;
      else if ((uint32_t)h.prim >= S.n_tris) cls = QC_LIGHT;  // a disk or sphere emitter
      else cls = class_of(__ldg(&S.mats[__ldg(&S.tri_info[h.prim].w)].type));
      w.cls_of[i] = (uint8_t)cls;
      ++traced;
    }
  }
  if (traced) atomicAdd(cnt64(w.cnt, CNT_SEGMENTS_LO), (unsigned long long)traced);
}


// Persistent closest-hit kernel with dynamic ray fetch: every warp keeps 32 rays in flight and,
// whenever at least `refill` of its lanes have finished (or the queue is drained and all have),
// hands the finished ones to the material queues and fetches new rays for the idle lanes with one
// atomic.  Traversal state (pt_scene.cuh TravState) is resumable, so lanes never wait for the
// slowest ray of a whole block (T. Aila, S. Laine, "Understanding the efficiency of ray traversal
// on GPUs", HPG 2009: persistent threads with ray replacement).
// kMulti: the rays belong to several scenes (a batch); each lane keeps its ray's scene view in
// registers.  Otherwise the single scene is the kernel parameter S0.
// kW4: the 4-wide BVH (node steps of pt_scene.cuh trav4_*, the next target `cur` a node, a leaf or
// kDone4); otherwise the BVH2 with the postponed-leaf pair (leafA, leafB).
template <bool kMulti, bool kW4>
__global__ void __launch_bounds__(kTraceBlock, PT_TRACE_MIN_BLOCKS) k_extend_persistent(SceneDev S0, WfDev w, int refill)
{
  __shared__ uint2 stk[(kW4 ? kRing4 : kShortStack) * kTraceBlock];
  const uint32_t n = w.cnt[w.in_slot];
  uint32_t* fetch = w.cnt + CNT_FETCH_EXT;
  TravGeom g = trav_geom(S0);
  float eps = S0.integ.scene_epsilon;
  const MatDev* mats = S0.mats;
  const int4* tinfo = S0.tri_info;
  const unsigned lane = threadIdx.x & 31;
  bool has = false, done = false, drained = false;
  uint32_t pid = 0, qi = 0, traced = 0;
  float3 o = f3s(0.0f), d = f3s(0.0f);
  std::conditional_t<kW4, RayPre4, RayPre> rp{};
  Hit h;
  h.t = 0.0f; h.u = h.v = 0.0f; h.prim = -1;
  TravState st;
  trav_init(st, stk + threadIdx.x, kTraceBlock);
  uint32_t leafA = 0, leafB = 0;
  uint2 spill4[kW4 ? kSpill4 : 1];
  Stack4 s4;
  stack4_init(s4, stk + threadIdx.x, kTraceBlock, spill4);
  int cur = kDone4;
  for (;;) {
    unsigned idle = __ballot_sync(0xffffffffu, !has);
    if (!drained && (__popc(idle) >= refill || idle == 0xffffffffu)) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, (uint32_t)__popc(idle));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + __popc(idle) >= n) drained = true;
      if (!has) {
        uint32_t i = base + __popc(idle & lanemask_lt());
        if (i < n) {
          pid = w.q_in[i];
          qi = i;
          if constexpr (kMulti) {
            const SceneDev& S = scene_of(w, pid);
            g = trav_geom(S);
            eps = S.integ.scene_epsilon;
            mats = S.mats;
            tinfo = S.tri_info;
          }
          float4 o4 = w.ray_o[pid], d4 = w.ray_d[pid];
          o = ld3(o4);
          d = ld3(d4);
          if constexpr (kW4) rp = ray_pre4(o, d, g.trav_scale);
          else rp = ray_pre(o, d, g.trav_scale);
          h.t = kDefaultMax;
          h.u = h.v = 0.0f;
          h.prim = -1;
          if constexpr (kW4) {
            stack4_init(s4, stk + threadIdx.x, kTraceBlock, spill4);
            cur = 0;
          } else {
            trav_init(st, stk + threadIdx.x, kTraceBlock);
          }
          has = true;
          done = false;
          ++traced;
        }
      }
    }
    if (__ballot_sync(0xffffffffu, has) == 0) break;
    for (;;) {
      // a warp-wide phase: intersect the postponed leaves (4-wide: when the lanes holding leaves are at
      // least kLeafVsNodeClosest times those that can take a node step; BVH2: at least as many), else
      // advance the lanes without leaves by one node
      if constexpr (kW4) {
        const bool lp = has && cur < 0;
        const bool np = has && cur >= 0 && cur != kDone4;
        const unsigned lmask = __ballot_sync(0xffffffffu, lp);
        const unsigned nmask = __ballot_sync(0xffffffffu, np);
        if (lmask && (nmask == 0 || __popc(lmask) >= kLeafVsNodeClosest * __popc(nmask))) {
          if (lp) {
            leaf_closest(g, (uint32_t)cur, o, d, eps, h);
            cur = stack4_next(s4, h.t, true);
          }
        } else if (np) {
          cur = trav4_node_closest(g, cur, rp, eps, h, s4);
        }
        done = cur == kDone4;
      } else {
        const bool lp = has && leafA != 0;
        const unsigned lmask = __ballot_sync(0xffffffffu, lp);
        const unsigned nmask = __ballot_sync(0xffffffffu, has && !done && !lp);
        if (lmask && (nmask == 0 || __popc(lmask) >= __popc(nmask))) {
          if (lp) {
            leaf_closest(g, leafA, o, d, eps, h);
            if (leafB) leaf_closest(g, leafB, o, d, eps, h);
            leafA = leafB = 0;
          }
        } else if (has && !done && !lp) {
          done = trav_node_closest(g, o, rp, eps, h, st, leafA, leafB);
        }
      }
      unsigned fin = __ballot_sync(0xffffffffu, !has || (done && leafA == 0));
      if (fin == 0xffffffffu || (!drained && __popc(fin) >= refill)) break;
    }
    int cls = -1;
    if (has && done && leafA == 0) {
      // the analytic emitters (disk and sphere lights) after the triangles
      uint32_t n_tris;
      if constexpr (kMulti) {
        const SceneDev& S = scene_of(w, pid);
        n_tris = S.n_tris;
        if (S.n_ana) ana_closest(S, o, d, eps, h);
      } else {
        n_tris = S0.n_tris;
        if (S0.n_ana) ana_closest(S0, o, d, eps, h);
      }
      w.hit[pid] = make_float4(h.t, h.u, h.v, as_float(h.prim));
      cls = h.prim < 0 ? QC_MISS : (uint32_t)h.prim >= n_tris ? QC_LIGHT : class_of(__ldg(&mats[__ldg(&tinfo[h.prim].w)].type));
      w.cls_of[qi] = (uint8_t)cls;
    }
    if (has && done && leafA == 0) has = false;
  }
  traced += __shfl_xor_sync(0xffffffffu, traced, 16);
  traced += __shfl_xor_sync(0xffffffffu, traced, 8);
  traced += __shfl_xor_sync(0xffffffffu, traced, 4);
  traced += __shfl_xor_sync(0xffffffffu, traced, 2);
  traced += __shfl_xor_sync(0xffffffffu, traced, 1);
  if (lane == 0 && traced) atomicAdd(cnt64(w.cnt, CNT_SEGMENTS_LO), (unsigned long long)traced);
}

// ------------------------------------------------------------------ binning by material (the sort by material key)
// The extend kernels record the class of the ray at each queue position (cls_of); these three kernels
// partition the queue stably by class into the material queues, so that each queue keeps the order of
// the rays it came from: camera rays in pixel order, later bounces in the order the shading kernels
// appended them.  Neighbouring entries of a material queue then address neighbouring path records
// (coalesced state reads and writes in the shading kernels) and emit spatially coherent shadow rays.
// The queue is cut into chunks of kBinThreads * kItems positions (kItems consecutive positions per
// thread; kItems = 4, 8 or 16, the launch option "bin_items" that the autotuner sets -- the sort
// granularity); k_bin_count counts every chunk's classes, k_bin_scan turns the counts into each
// chunk's start in every material queue (one block, chunk order), and k_bin_scatter writes every
// chunk's entries there.
constexpr int kBinThreads = 256;
constexpr int kBinItemsMin = 4;
constexpr int kBinWarps = kBinThreads / 32;
__host__ __device__ constexpr uint32_t bin_chunk(int items) { return (uint32_t)kBinThreads * (uint32_t)items; }

// The classes of the kItems positions of this thread in chunk k (-1 past the end of the queue); a full
// run is one aligned vector load of kItems bytes.
template <int kItems>
__device__ __forceinline__ void bin_load(const WfDev& w, uint32_t n, uint32_t k, int c[kItems])
{
  const uint32_t i0 = k * bin_chunk(kItems) + threadIdx.x * kItems;
  if (i0 + kItems <= n) {
    uint32_t v[kItems / 4];
    if constexpr (kItems == 4) {
      v[0] = *reinterpret_cast<const uint32_t*>(w.cls_of + i0);
    } else if constexpr (kItems == 8) {
      const uint2 u = *reinterpret_cast<const uint2*>(w.cls_of + i0);
      v[0] = u.x;
      v[1] = u.y;
    } else {
      const uint4 u = *reinterpret_cast<const uint4*>(w.cls_of + i0);
      v[0] = u.x;
      v[1] = u.y;
      v[2] = u.z;
      v[3] = u.w;
    }
#pragma unroll
    for (int j = 0; j < kItems; ++j) c[j] = (int)((v[j >> 2] >> (8 * (j & 3))) & 0xffu);
  } else {
#pragma unroll
    for (int j = 0; j < kItems; ++j) c[j] = i0 + j < n ? (int)w.cls_of[i0 + j] : -1;
  }
}

template <int kItems>
__global__ void __launch_bounds__(kBinThreads) k_bin_count(WfDev w)
{
  __shared__ uint32_t cnt[kQueues];
  const uint32_t n = w.cnt[w.in_slot];
  const uint32_t chunks = (n + bin_chunk(kItems) - 1) / bin_chunk(kItems);
  for (uint32_t k = blockIdx.x; k < chunks; k += gridDim.x) {
    if (threadIdx.x < kQueues) cnt[threadIdx.x] = 0;
    __syncthreads();
    int c[kItems];
    bin_load<kItems>(w, n, k, c);
#pragma unroll
    for (int q = 0; q < kQueues; ++q) {
      uint32_t v = 0;
#pragma unroll
      for (int j = 0; j < kItems; ++j) v += c[j] == q;
      for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if ((threadIdx.x & 31) == 0 && v) atomicAdd(&cnt[q], v);
    }
    __syncthreads();
    if (threadIdx.x < kQueues) w.bin[(size_t)k * kQueues + threadIdx.x] = cnt[threadIdx.x];
  }
}

// One block of 1024 threads per class q (blockIdx.x): the exclusive scan of the class's chunk counts
// (in place, chunk order) and its total (the material queue count).
__global__ void __launch_bounds__(1024) k_bin_scan(WfDev w, uint32_t chunk)
{
  __shared__ uint32_t warp_sum[32];
  const uint32_t n = w.cnt[w.in_slot];
  const uint32_t chunks = (n + chunk - 1) / chunk;
  const uint32_t per = (chunks + 1023) / 1024;  // consecutive chunks per thread
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  {
    const int q = blockIdx.x;
    uint32_t v = 0;
    for (uint32_t j = 0; j < per; ++j) {
      const uint32_t k = t * per + j;
      if (k < chunks) v += w.bin[(size_t)k * kQueues + q];
    }
    uint32_t x = v;  // inclusive warp scan of the per-thread sums
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
      uint32_t s = warp_sum[lane];
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, s, off);
        if (lane >= off) s += y;
      }
      warp_sum[lane] = s;
    }
    __syncthreads();
    uint32_t run = x - v + (wid ? warp_sum[wid - 1] : 0u);
    for (uint32_t j = 0; j < per; ++j) {
      const uint32_t k = t * per + j;
      if (k < chunks) {
        const uint32_t c = w.bin[(size_t)k * kQueues + q];
        w.bin[(size_t)k * kQueues + q] = run;
        run += c;
      }
    }
    if (t == 0) w.cnt[CNT_Q_MISS + q] = warp_sum[31];
  }
}

template <int kItems>
__global__ void __launch_bounds__(kBinThreads) k_bin_scatter(WfDev w)
{
  __shared__ uint32_t wtot[kBinWarps][kQueues];
  const uint32_t n = w.cnt[w.in_slot];
  const uint32_t chunks = (n + bin_chunk(kItems) - 1) / bin_chunk(kItems);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint32_t k = blockIdx.x; k < chunks; k += gridDim.x) {
    int c[kItems];
    bin_load<kItems>(w, n, k, c);
    uint32_t pos[kQueues];
#pragma unroll
    for (int q = 0; q < kQueues; ++q) {  // exclusive prefix of this thread's count over the warp
      uint32_t v = 0;
#pragma unroll
      for (int j = 0; j < kItems; ++j) v += c[j] == q;
      uint32_t x = v;
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
      }
      pos[q] = x - v;
      if (lane == 31) wtot[wid][q] = x;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kQueues; ++q) {
      uint32_t base = w.bin[(size_t)k * kQueues + q];
      for (int ww = 0; ww < wid; ++ww) base += wtot[ww][q];
      pos[q] += base;
    }
    const uint32_t i0 = k * bin_chunk(kItems) + threadIdx.x * kItems;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      if (c[j] < 0) continue;
      uint32_t at = 0;
#pragma unroll
      for (int q = 0; q < kQueues; ++q)
        if (c[j] == q) at = pos[q]++;
      w.q_mat[(size_t)c[j] * w.cap + at] = w.q_in[i0 + j];
    }
    __syncthreads();
  }
}

// The three binning launches at kItems positions per thread.
template <int kItems>
static void launch_binning(const WfDev& w, int grid, cudaStream_t st)
{
  k_bin_count<kItems><<<grid, kBinThreads, 0, st>>>(w);
  k_bin_scan<<<kQueues, 1024, 0, st>>>(w, bin_chunk(kItems));
  k_bin_scatter<kItems><<<grid, kBinThreads, 0, st>>>(w);
}

// Persistent any-hit kernel for the shadow queue (same ray replacement and BVH choice).
template <bool kMulti, bool kAdj, bool kW4>
__global__ void __launch_bounds__(kTraceBlock, PT_TRACE_MIN_BLOCKS) k_shadow_persistent(SceneDev S0, WfDev w, int refill)
{
  __shared__ uint2 stk[(kW4 ? kRing4 : kShortStack) * kTraceBlock];
  const uint32_t n = w.cnt[CNT_SHADOW];
  uint32_t* fetch = w.cnt + CNT_FETCH_SH;
  TravGeom g = trav_geom(S0);
  const unsigned lane = threadIdx.x & 31;
  bool has = false, drained = false, nodes_done = false;
  int res = 0;
  uint32_t slot = 0, leafA = 0, leafB = 0;
  float3 o = f3s(0.0f), d = f3s(0.0f);
  float tmin = 0.0f, tmax = 0.0f;
  std::conditional_t<kW4, RayPre4, RayPre> rp{};
  TravState st;
  trav_init(st, stk + threadIdx.x, kTraceBlock);
  uint2 spill4[kW4 ? kSpill4 : 1];
  Stack4 s4;
  stack4_init(s4, stk + threadIdx.x, kTraceBlock, spill4);
  int cur = kDone4;
  for (;;) {
    unsigned idle = __ballot_sync(0xffffffffu, !has);
    if (!drained && (__popc(idle) >= refill || idle == 0xffffffffu)) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, (uint32_t)__popc(idle));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + __popc(idle) >= n) drained = true;
      if (!has) {
        uint32_t i = base + __popc(idle & lanemask_lt());
        if (i < n) {
          slot = i;
          if constexpr (kMulti) g = trav_geom(scene_of(w, w.sh_pid[i]));
          float4 o4 = w.sh_o[i], d4 = w.sh_d[i];
          o = ld3(o4);
          d = ld3(d4);
          tmin = o4.w;
          tmax = d4.w;
          if constexpr (kW4) rp = ray_pre4(o, d, g.trav_scale);
          else rp = ray_pre(o, d, g.trav_scale);
          if constexpr (kW4) {
            stack4_init(s4, stk + threadIdx.x, kTraceBlock, spill4);
            cur = 0;
          } else {
            trav_init(st, stk + threadIdx.x, kTraceBlock);
          }
          has = true;
          res = 0;
          nodes_done = false;
          leafA = leafB = 0;
        }
      }
    }
    if (__ballot_sync(0xffffffffu, has) == 0) break;
    for (;;) {
      if constexpr (kW4) {
        const bool lp = has && res == 0 && cur < 0;
        const bool np = has && res == 0 && cur >= 0 && cur != kDone4;
        const unsigned lmask = __ballot_sync(0xffffffffu, lp);
        const unsigned nmask = __ballot_sync(0xffffffffu, np);
        if (lmask && (nmask == 0 || kLeafVsNodeAny * __popc(lmask) >= __popc(nmask))) {
          if (lp) {
            if (leaf_any(g, (uint32_t)cur, o, d, tmin, tmax)) res = 1;
            else cur = stack4_next(s4, tmax, false);
          }
        } else if (np) {
          cur = trav4_node_any(g, cur, rp, tmin, tmax, s4);
        }
        if (has && res == 0 && cur == kDone4) res = -1;
      } else {
        const bool lp = has && res == 0 && leafA != 0;
        const unsigned lmask = __ballot_sync(0xffffffffu, lp);
        const unsigned nmask = __ballot_sync(0xffffffffu, has && res == 0 && !nodes_done && !lp);
        if (lmask && (nmask == 0 || __popc(lmask) >= __popc(nmask))) {
          if (lp) {
            if (leaf_any(g, leafA, o, d, tmin, tmax) || (leafB && leaf_any(g, leafB, o, d, tmin, tmax))) res = 1;
            leafA = leafB = 0;
          }
        } else if (has && res == 0 && !nodes_done && !lp) {
          nodes_done = trav_node_any(g, o, rp, tmin, tmax, st, leafA, leafB);
        }
        if (has && res == 0 && nodes_done && leafA == 0) res = -1;
      }
      unsigned fin = __ballot_sync(0xffffffffu, !has || res != 0);
      if (fin == 0xffffffffu || (!drained && __popc(fin) >= refill)) break;
    }
    if (has && res != 0) {
      if (res < 0) {
        if constexpr (kMulti) {
          const SceneDev& S = scene_of(w, w.sh_pid[slot]);
          if (!(S.n_ana && ana_any(S, o, d, tmin, tmax))) shadow_unoccluded<kAdj>(S, w, slot, w.sh_pid[slot]);
        } else {
          if (!(S0.n_ana && ana_any(S0, o, d, tmin, tmax))) shadow_unoccluded<kAdj>(S0, w, slot, w.sh_pid[slot]);
        }
      }
      has = false;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && n) atomicAdd(cnt64(w.cnt, CNT_SHADOW_TOTAL), (unsigned long long)n);
}

// ------------------------------------------------------------------ shading kernels
// One kernel per material class: the vertices of pt_wavefront.cuh for every hit of the class's queue.
template <bool kAdj>
__global__ void __launch_bounds__(kBlock) k_shade_miss(WfDev w)
{
  const uint32_t n = w.cnt[CNT_Q_MISS];
  const uint32_t* q = w.q_mat + (size_t)QC_MISS * w.cap;
  for (uint32_t i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
    uint32_t pid = q[i];
    miss_path<kAdj>(scene_of(w, pid), w, pid);
  }
}

template <bool kAdj>
__global__ void __launch_bounds__(kBlock) k_shade_light(WfDev w)
{
  const uint32_t n = w.cnt[CNT_Q_LIGHT];
  const uint32_t* q = w.q_mat + (size_t)QC_LIGHT * w.cap;
  for (uint32_t i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
    uint32_t pid = q[i];
    light_path<kAdj>(scene_of(w, pid), w, pid);
  }
}

template <bool kAdj>
__global__ void __launch_bounds__(kBlock) k_shade_diffuse(WfDev w)
{
  __shared__ uint32_t sm[kWarps + 1];
  const uint32_t n = w.cnt[CNT_Q_DIFFUSE];
  const uint32_t* q = w.q_mat + (size_t)QC_DIFFUSE * w.cap;
  uint32_t clamped = 0;
  uint32_t overflow = 0;
  for (uint32_t base = blockIdx.x * kBlock; base < n; base += gridDim.x * kBlock) {
    uint32_t i = base + threadIdx.x;
    bool shadow = false, cont = false;
    uint32_t pid = 0;
    NeeRay nee;
    if (i < n) {
      pid = q[i];
      cont = diffuse_path<kAdj>(scene_of(w, pid), w, pid, nee, shadow, clamped, overflow);
    }
    uint32_t s_slot = block_slot(shadow, w.cnt + CNT_SHADOW, sm);
    if (shadow) {
      put_nee(w, s_slot, nee);
      w.sh_pid[s_slot] = pid;
    }
    uint32_t c_slot = block_slot(cont, w.cnt + w.out_slot, sm);
    if (cont) w.q_out[c_slot] = pid;
  }
  if (clamped) atomicAdd(cnt64(w.cnt, CNT_CLAMPED), (unsigned long long)clamped);
  if (overflow) atomicAdd(cnt64(w.cnt, CNT_ERROR), (unsigned long long)overflow);
}

// Paths with pending dipole gathers, appended to `out` (warp-aggregated).
__global__ void __launch_bounds__(kBlock) k_gather_collect(WfDev w, uint64_t n_paths, uint32_t* out)
{
  for (uint64_t base = (uint64_t)blockIdx.x * kBlock; base < n_paths; base += (uint64_t)gridDim.x * kBlock) {
    uint64_t pid = base + threadIdx.x;
    bool want = pid < n_paths && (w.rng[pid].w >> META_GSHIFT) != 0;
    unsigned m = __ballot_sync(0xffffffffu, want);
    if (m) {
      int leader = __ffs(m) - 1;
      uint32_t b = 0;
      if ((int)(threadIdx.x & 31) == leader) b = atomicAdd(w.cnt + CNT_GATHER, (uint32_t)__popc(m));
      b = __shfl_sync(0xffffffffu, b, leader);
      if (want) out[b + __popc(m & lanemask_lt())] = (uint32_t)pid;
    }
  }
}

// The dipole gathers of subsurface_scattering_shader.cu:126-173, evaluated for each path in the
// reverse order of their vertices (the post-order of the reference's recursion).  Per probe with
// L != 0 of the path's frame and object: distance Russian roulette with p = exp(-dist * min sigma_tr)
// on one MD5 draw, and on acceptance T12 * L * S(probe, xo) / p with the standard or directional
// dipole.  The sum times global_coeff / samples is added to the path's radiance, weighted by the
// throughput at the vertex.  The MD5 stream of a path is one sequential chain, so a lane owns a path.
//
// What bounds it: issue to the two integer pipes.  The 64 MD5 steps are a logic operation, a three-operand sum
// and a shift-and-add each: 190 ALU instructions per draw, 3.0 clocks of an SM at 64 lanes a clock, if all run
// there.  With the sums on the FMA pipe (md5_u2_split) they are 134 ALU and 128 FMA instructions: at least
// 2.1 clocks of either pipe, and 2.05 of the SM's four issue slots (128 lanes a clock).  The rest of a pair
// is kept out of the way:
//  * the roulette is decided from the draw's upper 31 bits against an upper bound of p taken with the
//    approximate square root and exponential (gather_bound); only the pairs that this bound cannot
//    reject (the accepted ones and about one in 10^4 more) go through the exact test, which alone
//    decides;
//  * those pairs are queued per warp in shared memory and evaluated 32 at a time, one pair per lane,
//    so that the dipole runs on full warps instead of on the lanes that happened to accept; a lane
//    then adds the values of its own pairs in probe order, so the sum is the sequential one bit for bit;
//  * a lane whose path is done takes the next path of the list at once, and the warp steps through the
//    pairs without any test of the lanes' ends until the first of them is due;
//  * the next probe is loaded before the draw and bounded after it.
// 456,028 gathers of 3,011 pairs (512 x 512 x 4 frames, 4,096 probes): 16.4 ms, 84.0 Gpair/s, 302 thread
// instructions a pair at 71 % of the issue slots, against 19.6 ms for one thread per path with the exact test in
// the probe loop and the dipole on the accepting lanes; gathers of few pairs and many acceptances take less than
// half of what they took so.  Six blocks per SM with the evaluation out of line: 5 blocks the same, 8 to 12
// spill and are 2 to 4 % slower.
//
// A differentiable forward render also stores each gather's value with the path (adj_G).  kAdj: the
// adjoint replays the same chain; a queued pair of a differentiated material adds the standard dipole's
// derivatives with respect to sigma_a and sigma_s' per channel (dipole_channel_grad) times its weight *
// L / p and its gather's factor (image gradient x throughput x global_coeff / samples) to the warp's sums
// for the material's gradient buffer (GatherGrad).
constexpr int kGatherQueue = 64;  // per warp; at most 31 + 32 entries are held
struct GatherWarp {
  uint4 q[kGatherQueue];   // queued pairs: owner lane, probe of its set, the draw's two words
  float4 xo[32];           // per owner lane, its current gather: position, min sigma_tr
  float4 f[32];            //   forward: boundary weight and rough flag; adjoint: factor
  float4 no[32];           //   forward: normal
  unsigned long long pb[32];  // first probe of the set
  uint2 sm[32];            //   scene of the pass, material
  float4 val[32];          // a flush's values and whether the pair was accepted
};

// Upper bound, scaled by 2^31, of the acceptance probability exp(-dist(p, xo) * chosen) with c2 = chosen
// * log2(e).  The approximate square root and exponential and the product's roundings are within 1e-5
// relative while the probability is above 2^-32; the slack is 1e-4 relative plus 5 * 2^-31.  A NaN
// anywhere gives NaN, which rejects nothing.
__device__ __forceinline__ float gather_bound(const float4& p, const float3& xo, float c2)
{
  const float dx = xo.x - p.x, dy = xo.y - p.y, dz = xo.z - p.z;
  const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
  float dist, e;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(dist) : "f"(d2));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(dist * -c2));
  return __fmaf_rn(e, 2147483648.0f * 1.0001f, 5.0f);
}

// Adjoint: what a warp has gathered for the gradient buffer `g` (6 floats), per lane.  A buffer takes
// one warp reduction and six atomics when the warp turns to another material's buffer and at its end:
// adding every flush's sum at once kept all warps waiting for the same six addresses.
struct GatherGrad {
  float* g = nullptr;
  float v[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
};
__device__ __forceinline__ void gather_grad_emit(GatherGrad& a, int lane)
{
  if (!a.g) return;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    float r = a.v[j];
    for (int off = 16; off; off >>= 1) r += __shfl_xor_sync(0xffffffffu, r, off);
    if (lane == 0) atomicAdd(a.g + j, r);
    a.v[j] = 0.0f;
  }
}

// One queued pair of the warp: its value (forward: the term with its weight; adjoint: d / d sigma_a and
// d / d sigma_s') where the exact test accepts it.  Out of line, so that the probe loop keeps its registers.
struct GatherValue {
  float3 v, ds;
  int ok;
};
template <bool kAdj>
static __device__ __noinline__ GatherValue gather_eval(const SceneDev* scenes, const float4* pc_pos, const float4* pc_wl, const float4* pc_nrm,
                                                       const float4* pc_tr, const GatherWarp* sp, int lane)
{
  const GatherWarp& s = *sp;
  GatherValue r{f3s(0.0f), f3s(0.0f), 0};
  const uint4 e = s.q[lane];
  const uint32_t o = e.x;
  const float4 x4 = s.xo[o], f4 = s.f[o];
  const uint2 id = s.sm[o];
  const SceneDev& S = scenes[id.x];
  const ScatDev& P = S.scat[id.y];
  const uint64_t at = s.pb[o] + e.y;
  const float3 xo = ld3(x4);
  const float3 pos = ld3(__ldg(pc_pos + at));
  const float dist = length(xo - pos);
  const float exp_term = expf(-dist * x4.w);
  const float rn = md5_draw(e.z, e.w);
  if constexpr (kAdj) {
    if (rn < exp_term) {
      const float scale = S.mats[id.y].a.x;
      const float3 wl = ld3(__ldg(pc_wl + at));
      const Dual2 sx = dipole_channel_grad(dist, P.absorption.x, P.reducedExtinction.x, P.A.x, scale);
      const Dual2 sy = dipole_channel_grad(dist, P.absorption.y, P.reducedExtinction.y, P.A.y, scale);
      const Dual2 sz = dipole_channel_grad(dist, P.absorption.z, P.reducedExtinction.z, P.A.z, scale);
      const float3 k = ld3(f4) * wl / exp_term;
      r.v = k * f3(sx.da, sy.da, sz.da);
      r.ds = k * f3(sx.ds, sy.ds, sz.ds);
      r.ok = 1;
    }
  } else {
    const bool rough = f4.w != 0.0f;  // rough boundary: draws must exceed 0.001, terms carry the weight
    if (rn < exp_term && (!rough || rn > 0.001f)) {
      const float3 wl = ld3(__ldg(pc_wl + at));
      float3 term;
      if (S.mats[id.y].model == DIRECTIONAL_DIPOLE)
        term = wl * dirpole_bssrdf(pos, ld3(__ldg(pc_nrm + at)), ld3(__ldg(pc_tr + at)), xo, ld3(s.no[o]), P) / exp_term;
      else
        term = wl * dipole_bssrdf(dist, std_dipole_terms(P)) / exp_term;
      r.v = rough ? term * ld3(f4) : term;
      r.ok = 1;
    }
  }
  return r;
}

// Evaluates the first `count` queued pairs of the warp, one per lane.  Forward: adds the values of the
// calling lane's own pairs (bits of `mine`, queue order = probe order) to acc.  Adjoint: adds the pair's
// derivatives to grad.
template <bool kAdj>
__device__ __forceinline__ void gather_flush(const WfDev& w, const SssDev& g, GatherWarp& s, int count, int lane, unsigned mine, float3& acc,
                                             GatherGrad& grad)
{
  __syncwarp();
  GatherValue e{f3s(0.0f), f3s(0.0f), 0};
  if (lane < count) e = gather_eval<kAdj>(w.scenes, g.pc_pos, g.pc_wl, g.pc_nrm, g.pc_tr, &s, lane);
  __syncwarp();
  if constexpr (kAdj) {
    float* gr = nullptr;
    if (e.ok) {
      const uint2 id = s.sm[s.q[lane].x];
      gr = w.scenes[id.x].mat_grad[id.y];
    }
    const unsigned have = __ballot_sync(0xffffffffu, gr != nullptr);
    if (have == 0) return;
    const unsigned long long g0 = __shfl_sync(0xffffffffu, (unsigned long long)gr, __ffs(have) - 1);
    if (__all_sync(0xffffffffu, gr == nullptr || (unsigned long long)gr == g0)) {
      if ((unsigned long long)grad.g != g0) {
        gather_grad_emit(grad, lane);
        grad.g = (float*)g0;
      }
      grad.v[0] += e.v.x;
      grad.v[1] += e.v.y;
      grad.v[2] += e.v.z;
      grad.v[3] += e.ds.x;
      grad.v[4] += e.ds.y;
      grad.v[5] += e.ds.z;
    } else if (gr) {
      atomicAdd(gr + 0, e.v.x);
      atomicAdd(gr + 1, e.v.y);
      atomicAdd(gr + 2, e.v.z);
      atomicAdd(gr + 3, e.ds.x);
      atomicAdd(gr + 4, e.ds.y);
      atomicAdd(gr + 5, e.ds.z);
    }
  } else {
    s.val[lane] = make_float4(e.v.x, e.v.y, e.v.z, e.ok ? 1.0f : 0.0f);
    __syncwarp();
    for (; mine; mine &= mine - 1) {
      const float4 t = s.val[__ffs(mine) - 1];
      if (t.w != 0.0f) acc = acc + ld3(t);
    }
  }
}

template <bool kAdj>
__global__ void __launch_bounds__(kBlock, 6) k_gather(WfDev w, SssDev g, const uint32_t* list, uint32_t one)
{
  __shared__ GatherWarp shared[kWarps];
  const uint32_t n = w.cnt[CNT_GATHER];
  const int lane = threadIdx.x & 31;
  GatherWarp& s = shared[threadIdx.x >> 5];
  int qn = 0;                     // queued pairs (warp-uniform)
  unsigned long long mine = 0;    // this lane's among them
  unsigned long long pairs = 0, gathers = 0;
  bool active = true, in_gather = false;
  int slot = -1;                  // gathers of the path left below the current one
  uint32_t pid = 0xffffffffu, k = 0, nc = 0;
  uint2 t64 = make_uint2(0, 0);
  float3 xo = f3s(0.0f), acc = f3s(0.0f);
  float c2 = 0.0f, bound = 0.0f;
  const float4* probes = g.pc_pos;
  GatherGrad grad;
  for (;;) {
    // lanes at the end of a gather: its pending pairs, its sum, and the next gather of the path or the
    // next path of the list
    const bool end = active && k >= nc;
    if (__any_sync(0xffffffffu, end && mine != 0)) {
      // The probe loop leaves at most 31 pairs queued, so this drains the queue in one round.  It stays a loop:
      // the kernel compiled with a plain flush here is the same within 1 % for many gathers but loses 20 % where a
      // few are bound by their draws' latency (203 x 151, 500 probes: 680 us a frame against 815 to 890).
      for (; qn > 0; qn -= 32) gather_flush<kAdj>(w, g, s, qn, lane, (unsigned)mine, acc, grad);
      mine = 0;
      qn = 0;
    }
    if (end) {
      for (;;) {
        const ItemDev* it = nullptr;
        const SceneDev* S = nullptr;
        uint32_t fl = 0;
        if (pid != 0xffffffffu) {
          it = &w.items[w.path_item[pid]];
          S = &w.scenes[it->scene];
          fl = (uint32_t)((pid - it->path_begin) / it->pixels);
        }
        if (in_gather) {
          in_gather = false;
          if constexpr (!kAdj) {
            const size_t at = (size_t)(slot + 1) * w.cap + pid;
            const float3 thr = f3(w.g_a[at].w, w.g_b[at].w, w.g_c[at].x);
            const float3 contrib = acc * S->scat[__float_as_int(w.g_c[at].y)].global_coeff / (float)S->probe_samples;
            const float4 r = w.rad[pid];
            const float3 L = ld3(r) + thr * contrib;
            w.rad[pid] = make_float4(L.x, L.y, L.z, r.w);
            if (S->adj_G) {
              const uint64_t gp = (uint64_t)(it->first_frame + fl - S->adj_first) * it->pixels + (pid - it->path_begin) % it->pixels;
              S->adj_G[gp * S->adj_slots + slot + 1] = make_float4(contrib.x, contrib.y, contrib.z, 0.0f);
            }
          }
        }
        if (slot < 0) {
          if (pid != 0xffffffffu) {
            const uint4 rg = w.rng[pid];
            w.rng[pid] = make_uint4(rg.x, t64.x, t64.y, rg.w);
          }
          const uint32_t i = atomicAdd(w.cnt + CNT_FETCH_GATHER, 1u);
          if (i >= n) {
            active = false;
            pid = 0xffffffffu;
            break;
          }
          pid = list[i];
          const uint4 rg = w.rng[pid];
          t64 = make_uint2(rg.y, rg.z);
          slot = (int)(rg.w >> META_GSHIFT) - 1;
          continue;
        }
        const size_t at = (size_t)slot * w.cap + pid;
        --slot;
        const float4 a = w.g_a[at];
        const int mat = __float_as_int(w.g_c[at].y);
        if (mat < 0) {  // reset marker: the MD5 state the vertex below was entered with
          t64 = make_uint2(__float_as_uint(a.x), __float_as_uint(a.y));
          continue;
        }
        const ScatDev& P = S->scat[mat];
        const uint32_t set_in_item = fl * S->n_trans + S->mats[mat].aux;
        const uint64_t pb = it->probe_begin + (uint64_t)set_in_item * S->probe_samples;
        const float chosen = fminf(P.transport.x, fminf(P.transport.y, P.transport.z));
        nc = g.pc_cnt[it->set_begin + set_in_item];
        k = 0;
        acc = f3s(0.0f);
        in_gather = true;
        pairs += nc;
        ++gathers;
        if (nc == 0) continue;
        xo = ld3(a);
        c2 = chosen * 1.44269504f;
        probes = g.pc_pos + pb;
        s.xo[lane] = make_float4(xo.x, xo.y, xo.z, chosen);
        s.pb[lane] = pb;
        s.sm[lane] = make_uint2(it->scene, (uint32_t)mat);
        bound = gather_bound(__ldg(probes), xo, c2);
        if constexpr (kAdj) {
          const float3 thr = f3(a.w, w.g_b[at].w, w.g_c[at].x);
          const float3 f = ld3(w.adj_a[pid]) * thr * P.global_coeff / (float)S->probe_samples;
          s.f[lane] = make_float4(f.x, f.y, f.z, S->mat_grad[mat] ? 1.0f : 0.0f);
        } else {
          s.f[lane] = w.g_d[at];
          s.no[lane] = w.g_b[at];
        }
        break;
      }
    }
    if (!__any_sync(0xffffffffu, active)) break;
    // the adjoint queues the pairs of differentiated materials only
    const bool take = active && (!kAdj || s.f[lane].w != 0.0f);
    const uint32_t step = active ? 1u : 0u;
    for (uint32_t rem = __reduce_min_sync(0xffffffffu, active ? nc - k : 0xffffffffu); rem; --rem) {
      const float4 next = __ldg(probes + (k + step));
      uint32_t h0, h1;
      md5_u2_split(t64.x, t64.y, one, h0, h1);
      t64 = make_uint2(h0, h1);
      const bool cand = take && !((float)(int)(h1 & 0x7fffffffu) > bound);
      const unsigned m = __ballot_sync(0xffffffffu, cand);
      if (m) {
        if (cand) {
          const int at = qn + __popc(m & lanemask_lt());
          s.q[at] = make_uint4((uint32_t)lane, k, h0, h1);
          mine |= 1ull << at;
        }
        qn += __popc(m);
        if (qn >= 32) {
          gather_flush<kAdj>(w, g, s, 32, lane, (unsigned)mine, acc, grad);
          mine >>= 32;
          qn -= 32;
          uint4 moved = make_uint4(0, 0, 0, 0);
          if (lane < qn) moved = s.q[32 + lane];
          __syncwarp();
          if (lane < qn) s.q[lane] = moved;
        }
      }
      bound = gather_bound(next, xo, c2);
      k += step;
    }
  }
  if constexpr (kAdj) gather_grad_emit(grad, lane);
  if (pairs) atomicAdd(cnt64(w.cnt, CNT_PAIRS), pairs);
  if (gathers) atomicAdd(cnt64(w.cnt, CNT_GATHERS), gathers);
}

// sample_camera.cu:48-268 for a smooth translucent object, with GLOBAL and RND_64 defined: probe j of
// the group (frame-major, then object, then sample; path id j - j0).  The triangle is picked with an
// MD5 draw, the point uniformly on it, and with probability 1/2 (one LCG draw) the probe is lit by a
// light sample with a shadow ray (written to the path's radiance here), else by an indirect path
// started into the wavefront from the point (depth 0, emission on).  The record keeps pos, dir (of the
// light sample), normal, transmitted direction and T12; pad = (triangles * area, indirect flag) until
// k_probe_finish forms L.
__global__ void __launch_bounds__(kBlock) k_probe_gen(WfDev w, SssDev g, uint64_t j0, uint64_t n)
{
  __shared__ uint32_t sm[kWarps + 1];
  uint32_t clamped = 0;
  for (uint64_t base = (uint64_t)blockIdx.x * kBlock; base < n; base += (uint64_t)gridDim.x * kBlock) {
    uint64_t pid = base + threadIdx.x;
    bool indirect = false;
    if (pid < n) {
      uint64_t j = j0 + pid;
      uint32_t item = find_item(w.items, w.n_items, j, [](const ItemDev& x) { return x.probe_begin; });
      const ItemDev& it = w.items[item];
      const SceneDev& S = w.scenes[it.scene];
      const uint64_t per_frame = (uint64_t)S.n_trans * S.probe_samples;
      uint32_t fl = (uint32_t)((j - it.probe_begin) / per_frame);
      uint32_t idx = (uint32_t)((j - it.probe_begin) % per_frame);  // launch_index + current_translucent_obj * samples
      uint32_t k = idx / S.probe_samples;
      uint32_t frame = it.first_frame + fl;
      uint4 ob = S.trans_objs[k];
      const uint32_t triangles = ob.z;
      const ScatDev& P = S.scat[ob.x];
      uint32_t t = tea16(idx, frame);
      uint32_t s2 = tea16(idx, frame);
      uint2 t64 = make_uint2(s2, s2);
      uint32_t tid = (uint32_t)(int)(rnd_md5(t64) * (float)triangles);
      if (tid >= triangles) { tid = triangles - 1; ++clamped; }
      const float* v = S.trans_pos + 9 * ((size_t)ob.w + tid);
      float3 v0 = f3(v[0], v[1], v[2]), v1 = f3(v[3], v[4], v[5]), v2 = f3(v[6], v[7], v[8]);
      float3 perp = cross(v1 - v0, v2 - v0);
      float area = 0.5f * length(perp);
      float xi1 = sqrtf(rnd_md5(t64));
      float xi2 = rnd_md5(t64);
      float u = 1.0f - xi1, vv = (1.0f - xi2) * xi1, ww = xi1 * xi2;
      float3 pos = u * v0 + vv * v1 + ww * v2;
      int4 info = __ldg(S.tri_info + ob.y + tid);
      float3 nrm;
      if (info.x >= 0) {
        float3 n0 = ld3(__ldg(S.normals + info.x)), n1 = ld3(__ldg(S.normals + info.y)), n2 = ld3(__ldg(S.normals + info.z));
        nrm = normalize(u * n0 + vv * n1 + ww * n2);
        nrm = normalize(nrm);
      } else {
        nrm = normalize(perp);
      }
      const float recip_ior = 1.0f / P.relative_ior;
      // rough objects: the probe's normal is a microfacet normal sampled with two MD5 draws (:130-151)
      const MatDev& om = S.mats[ob.x];
      const bool rough = om.type == MAT_ROUGH_TRANSLUCENT;
      const float r_ax = om.a.y, r_ay = om.a.z;
      const uint32_t r_model = __float_as_uint(om.a.w), r_dist = om.dist;
      float3 mnorm = nrm;
      int capped = 0;
      auto microfacet = [&](const float3& wdir) {
        const float z1 = rnd_md5(t64);
        const float z2 = rnd_md5(t64);
        mnorm = r_model == WALTER ? sample_normal(r_dist, nrm, z1, z2, r_ax) : sample_visible_normal(r_dist, wdir, nrm, r_ax, r_ay, z1, z2, &capped);
      };
      float3 Le, w_i, dir = f3s(0.0f);
      if (rnd_lcg(t) < 0.5f) {
        uint32_t li = (uint32_t)((float)S.n_lights * rnd_md5(t64));
        if (li >= (uint32_t)S.n_lights) { li = (uint32_t)S.n_lights - 1; ++clamped; }
        float light_pdf = 1.0f / (float)S.n_lights;
        LightRaw ls = S.lights[li];
        float r = 0.0f;
        eval_direct(S, pos, ls, w_i, Le, r, t, clamped);
        dir = w_i;
        if (rough) microfacet(w_i);
        float cos_i = fmaxf(dot(w_i, nrm), 0.0f);
        if (cos_i > 0.0f) {
          float att = occluded(S, pos, w_i, S.integ.scene_epsilon, r) ? 0.0f : 1.0f;
          Le = Le * (att * cos_i / light_pdf);
        } else {
          Le = f3s(0.0f);
        }
        w.rad[pid] = make_float4(Le.x, Le.y, Le.z, 0.0f);
      } else {
        w_i = sample_cosine_weighted(nrm, t);
        if (rough) microfacet(w_i);
        w.ray_o[pid] = make_float4(pos.x, pos.y, pos.z, 0.0f);
        w.ray_d[pid] = make_float4(w_i.x, w_i.y, w_i.z, 0.0f);
        w.thr[pid] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
        w.rad[pid] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        w.rng[pid] = make_uint4(t, t64.x, t64.y, META_EMIT | META_PROBE);
        w.path_item[pid] = (uint16_t)item;
        indirect = true;
      }
      float cos_i = fmaxf(dot(w_i, mnorm), 0.0f);
      float cos_i2 = cos_i * cos_i;
      float st2 = recip_ior * recip_ior * (1.0f - cos_i2);
      float cos_t = sqrtf(1.0f - st2);
      float3 tr = recip_ior * (cos_i * mnorm - w_i) - mnorm * cos_t;
      float T12 = 1.0f - fresnel_R(cos_i, cos_t, recip_ior);
      float wgt = T12;  // 1 * T12
      if (rough) {  // :232-266
        if (r_model == WALTER) {
          const float G_i_m = masking_G1_aniso(r_dist, w_i, mnorm, nrm, r_ax, r_ay);
          const float abs_i_m = fabsf(dot(w_i, mnorm)), abs_i_n = fabsf(dot(w_i, nrm)), abs_n_m = fabsf(dot(nrm, mnorm));
          const float G_o_m = masking_G1_aniso(r_dist, tr, mnorm, nrm, r_ax, r_ay);
          wgt = (1.0f * (abs_i_m * G_i_m / (abs_i_n * abs_n_m) * G_o_m)) * T12;
        } else if (r_model == VISIBLE_NORMALS) {
          wgt = (1.0f * masking_G1_aniso(r_dist, tr, mnorm, nrm, r_ax, r_ay)) * T12;
        }
      }
      if (capped) atomicAdd(cnt64(w.cnt, CNT_CAPPED), 1ull);
      float4* rec = g.probes + 5 * j;
      rec[0] = make_float4(pos.x, pos.y, pos.z, dir.x);
      rec[1] = make_float4(dir.y, dir.z, mnorm.x, mnorm.y);
      rec[2] = make_float4(mnorm.z, 0.0f, 0.0f, 0.0f);
      rec[3] = make_float4(tr.x, tr.y, tr.z, wgt);
      rec[4] = make_float4(wgt, wgt, (float)triangles * area, indirect ? 1.0f : 0.0f);
    }
    uint32_t slot = block_slot(indirect, w.cnt + w.in_slot, sm);
    if (indirect) w.q_in[slot] = (uint32_t)pid;
  }
  if (clamped) atomicAdd(cnt64(w.cnt, CNT_CLAMPED), (unsigned long long)clamped);
}

// sample_camera.cu:207 and :230: Le = (light sample, or the indirect path's radiance times pi) / 0.5,
// L = Le * (triangles * area).
__global__ void __launch_bounds__(kBlock) k_probe_finish(WfDev w, SssDev g, uint64_t j0, uint64_t n)
{
  for (uint64_t pid = (uint64_t)blockIdx.x * kBlock + threadIdx.x; pid < n; pid += (uint64_t)gridDim.x * kBlock) {
    float4* rec = g.probes + 5 * (j0 + pid);
    float4 r4 = rec[4];
    float3 Le = ld3(w.rad[pid]);
    if (r4.w != 0.0f) Le = Le * kPi;
    Le = Le / 0.5f;
    float3 L = Le * r4.z;
    float4 r2 = rec[2];
    rec[2] = make_float4(r2.x, L.x, L.y, L.z);
    rec[4] = make_float4(r4.x, r4.y, 0.0f, 0.0f);
  }
}

// The probes with dot(L, L) > 0 of one (frame, object) set, compacted in order: one block per set.
__global__ void __launch_bounds__(256) k_probe_compact(WfDev w, SssDev g)
{
  __shared__ uint32_t warp_off[8];
  __shared__ uint32_t total;
  const uint32_t set = blockIdx.x;
  const ItemDev& it = w.items[find_item(w.items, w.n_items, set, [](const ItemDev& x) { return x.set_begin; })];
  const uint32_t samples = w.scenes[it.scene].probe_samples;
  const size_t b = it.probe_begin + (size_t)(set - it.set_begin) * samples;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t c0 = 0; c0 < samples; c0 += 256) {
    uint32_t i = c0 + threadIdx.x;
    bool keep = false;
    float3 pos, nrm, L, tr, wt;
    if (i < samples) {
      const float4* rec = g.probes + 5 * (b + i);
      float4 r0 = rec[0], r1 = rec[1], r2 = rec[2], r3 = rec[3], r4 = rec[4];
      pos = ld3(r0);
      nrm = f3(r1.z, r1.w, r2.x);
      L = f3(r2.y, r2.z, r2.w);
      tr = ld3(r3);
      wt = f3(r3.w, r4.x, r4.y);
      keep = dot(L, L) > 0.0f;
    }
    unsigned m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) warp_off[warp] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t run = total;
      for (int k = 0; k < 8; ++k) {
        uint32_t cnt = warp_off[k];
        warp_off[k] = run;
        run += cnt;
      }
      total = run;
    }
    __syncthreads();
    if (keep) {
      size_t o = b + warp_off[warp] + __popc(m & lanemask_lt());
      float3 wl = wt * L;
      g.pc_pos[o] = make_float4(pos.x, pos.y, pos.z, 0.0f);
      g.pc_wl[o] = make_float4(wl.x, wl.y, wl.z, 0.0f);
      g.pc_nrm[o] = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
      g.pc_tr[o] = make_float4(tr.x, tr.y, tr.z, 0.0f);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) g.pc_cnt[set] = total;
}

// Shadow rays of diffuse_shader.cu:69-81 (every material's any-hit program is opaque).
template <bool kAdj>
__global__ void __launch_bounds__(kBlock) k_shadow(WfDev w)
{
  const uint32_t n = w.cnt[CNT_SHADOW];
  for (uint32_t i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
    float4 o = w.sh_o[i], d = w.sh_d[i];
    uint32_t pid = w.sh_pid[i];
    const SceneDev& S = scene_of(w, pid);
    if (!scene_any(S, ld3(o), ld3(d), o.w, d.w)) shadow_unoccluded<kAdj>(S, w, i, pid);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && n) atomicAdd(cnt64(w.cnt, CNT_SHADOW_TOTAL), (unsigned long long)n);
}

// path_tracer.cu:36-43 and :64-68, frame by frame in order.
// One thread per (item, pixel): the item's frames are folded into the scene's running mean in order.
__global__ void __launch_bounds__(kBlock) k_accumulate(WfDev w, uint64_t n_pix)
{
  for (uint64_t q = (uint64_t)blockIdx.x * kBlock + threadIdx.x; q < n_pix; q += (uint64_t)gridDim.x * kBlock) {
    const ItemDev& it = w.items[find_item(w.items, w.n_items, q, [](const ItemDev& x) { return x.pix_begin; })];
    const uint32_t p = (uint32_t)(q - it.pix_begin);
    const SceneDev& S = w.scenes[it.scene];
    float4* accum = S.accum;
    float4 out = accum[p];
    for (uint32_t fl = 0; fl < it.n_frames; ++fl) {
      uint64_t pid = it.path_begin + (uint64_t)fl * it.pixels + p;
      uint32_t frame = it.first_frame + fl;
      if (S.adj_L) S.adj_L[(uint64_t)(frame - S.adj_first) * it.pixels + p] = w.rad[pid];
      if (w.rng[pid].w & META_OUTSIDE) {
        out = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        continue;
      }
      float4 r = w.rad[pid];
      if (isfinite(r.x) && isfinite(r.y) && isfinite(r.z)) {
        float4 cur = frame != 0 ? make_float4(out.x * (float)frame, out.y * (float)frame, out.z * (float)frame, out.w * (float)frame)
                                : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float den = (float)(frame + 1);
        out = make_float4((r.x + cur.x) / den, (r.y + cur.y) / den, (r.z + cur.z) / den, (1.0f + cur.w) / den);
      }
    }
    accum[p] = out;
  }
}

// Geometric normals (unnormalised cross(v1-v0, v2-v0)) per original triangle, for meshes without
// vertex normals and for the emitter test.
__global__ void k_geo_normals(SceneDev S, float4* geo)
{
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < S.n_tris; j += gridDim.x * blockDim.x) {
    float4 a = S.tri_v0[j], b = S.tri_e1[j], c = S.tri_e2[j];
    float3 n = cross(ld3(b), ld3(c));
    geo[__float_as_int(a.w)] = make_float4(n.x, n.y, n.z, 0.0f);
  }
}

// Probe paths of a chunk that may run beside its camera paths: 39 MB of wavefront at most.
constexpr uint64_t kProbesBesideMax = 1ull << 18;
static_assert(kCounters * 4 <= kProbeCounterBytes, "the probe wavefront's counters");
static pt_status ensure_probe_wavefront(ProbeWavefront& p, uint64_t cap)
{
  if (p.cap >= cap && p.buf.p) return PT_OK;
  p.cap = 0;
  const uint64_t n = (cap + 7) / 8 * 8;  // every array starts on a 16-byte boundary
  pt_status st = p.buf.reserve(kProbeCounterBytes + n * kProbePathBytes, "probe wavefront");
  if (st == PT_OK) p.cap = n;
  return st;
}
// Its device view: the arrays that the pools and the probe kernels read; the others stay as they are in v.
static void probe_view(const ProbeWavefront& p, WfDev& v)
{
  char* at = p.buf.as<char>();
  auto take = [&](size_t bytes) {
    char* r = at;
    at += bytes;
    return r;
  };
  v.cap = p.cap;
  v.cnt = reinterpret_cast<uint32_t*>(take(kProbeCounterBytes));
  float4* rays = reinterpret_cast<float4*>(take(p.cap * 32));
  float4* state = reinterpret_cast<float4*>(take(p.cap * 32));
  v.ray_o = Field2<float4>{rays};
  v.ray_d = Field2<float4>{rays + 1};
  v.thr = Field2<float4>{state};
  v.rng = Field2<uint4>{reinterpret_cast<uint4*>(state + 1)};
  for (float4** f : {&v.rad, &v.hit, &v.sh_o, &v.sh_d, &v.sh_c}) *f = reinterpret_cast<float4*>(take(p.cap * 16));
  v.q_in = reinterpret_cast<uint32_t*>(take(p.cap * 4));
  v.path_item = reinterpret_cast<uint16_t*>(take(p.cap * 2));
  v.q_out = v.q_mat = v.bin = v.sh_pid = nullptr;
  v.cls_of = nullptr;
  v.g_a = v.g_b = v.g_d = v.adj_a = v.adj_b = nullptr;
  v.g_c = nullptr;
  v.g_slots = 0;
}

static pt_status ensure_wavefront(Wavefront& wf, uint64_t cap)
{
  if (wf.cap >= cap && wf.counters.p) return PT_OK;
  pt_status st = PT_OK;
  const size_t f4 = sizeof(float4), u4 = sizeof(uint4);
  if (st == PT_OK) st = wf.rays.reserve(cap * 2 * f4, "wavefront ray records");
  if (st == PT_OK) st = wf.state.reserve(cap * (f4 + u4), "wavefront path-state records");
  if (st == PT_OK) st = wf.rad.reserve(cap * f4, "wavefront radiance");
  if (st == PT_OK) st = wf.hit.reserve(cap * f4, "wavefront hits");
  if (st == PT_OK) st = wf.path_item.reserve(cap * 2, "wavefront path items");
  if (st == PT_OK) st = wf.q_a.reserve(cap * 4, "queue");
  if (st == PT_OK) st = wf.q_b.reserve(cap * 4, "queue");
  if (st == PT_OK) st = wf.q_mat.reserve(cap * 4 * kQueues, "material queues");
  if (st == PT_OK) st = wf.cls_of.reserve(cap, "material classes of the queue");
  if (st == PT_OK) st = wf.bin.reserve(((cap + bin_chunk(kBinItemsMin) - 1) / bin_chunk(kBinItemsMin)) * kQueues * 4, "material binning counts");
  if (st == PT_OK) st = wf.sh_o.reserve(cap * f4, "shadow queue");
  if (st == PT_OK) st = wf.sh_d.reserve(cap * f4, "shadow queue");
  if (st == PT_OK) st = wf.sh_c.reserve(cap * f4, "shadow queue");
  if (st == PT_OK) st = wf.sh_pid.reserve(cap * 4, "shadow queue");
  if (st == PT_OK) st = wf.counters.reserve(kCounters * 4, "counters");
  if (st != PT_OK) {
    wf.cap = 0;
    return st;
  }
  wf.cap = cap;
  return PT_OK;
}

// Gather stacks for `cap` paths with `slots` entries each, and probe storage for `records` probes.
static pt_status ensure_sss(Context& c, uint64_t cap, uint32_t slots, uint64_t records, uint64_t sets)
{
  Wavefront& wf = c.wf;
  pt_status st = PT_OK;
  if (wf.gather_cap < cap || wf.gather_slots < slots || !wf.g_a.p) {
    const size_t n = (size_t)cap * slots;
    st = wf.g_a.reserve(n * sizeof(float4), "dipole gather stack");
    if (st == PT_OK) st = wf.g_b.reserve(n * sizeof(float4), "dipole gather stack");
    if (st == PT_OK) st = wf.g_c.reserve(n * sizeof(float2), "dipole gather stack");
    if (st == PT_OK) st = wf.g_d.reserve(n * sizeof(float4), "dipole gather stack");
    if (st != PT_OK) {
      wf.gather_cap = 0;
      wf.gather_slots = 0;
      return st;
    }
    wf.gather_cap = cap;
    wf.gather_slots = slots;
  }
  if (wf.probe_cap < records || !wf.probes.p) {
    st = wf.probes.reserve(records * 80, "probe records");
    // one position more than there are probes: the gathers load the probe after the one they draw for
    if (st == PT_OK) st = wf.pc_pos.reserve((records + 1) * sizeof(float4), "compacted probes");
    if (st == PT_OK) st = wf.pc_wl.reserve(records * sizeof(float4), "compacted probes");
    if (st == PT_OK) st = wf.pc_nrm.reserve(records * sizeof(float4), "compacted probes");
    if (st == PT_OK) st = wf.pc_tr.reserve(records * sizeof(float4), "compacted probes");
    if (st != PT_OK) {
      wf.probe_cap = 0;
      return st;
    }
    wf.probe_cap = records;
  }
  return wf.pc_cnt.reserve(std::max<uint64_t>(sets, 1) * 4, "probe counts");
}

static int __float_as_int_host(float f)
{
  int i;
  memcpy(&i, &f, 4);
  return i;
}

// Checks a scene before it is rendered and brings its device state up to date on its own stream:
// changed materials, and the geometric normals (once per build).
pt_status prepare_scene(Context& c, const char* who)
{
  PT_CHECK_CUDA(cudaSetDevice(c.device), "cudaSetDevice");
  if (!c.built) return fail(PT_NOT_READY, std::string(who) + ": call pt_build first");
  if (!c.camera_set) return fail(PT_NOT_READY, std::string(who) + ": camera not set");
  for (const LightRaw& l : c.lights)
    if (l.type == ENVMAP_LIGHT && !c.env_present) return fail(PT_NOT_READY, std::string(who) + ": an environment-map light needs pt_set_envmap");
  for (const MatDev& m : c.mats)
    if ((m.type == MAT_DIFFUSE || m.type == MAT_LAMBERTIAN_INTERFACE || m.type == MAT_ROUGH_DIFFUSE) && c.lights.empty())
      return fail(PT_NOT_READY, std::string(who) +
                                    ": diffuse materials need at least one light (light_buffer is indexed unguarded by the diffuse, "
                                    "lambertian-interface and rough-diffuse shaders)");
  const bool sss = !c.trans_objs.empty();
  if (sss && c.lights.empty())
    return fail(PT_NOT_READY, std::string(who) + ": translucent objects need at least one light (the probe pass samples light_buffer)");
  if (sss && c.integ.max_depth > 254)
    return fail(PT_CAP_EXCEEDED, std::string(who) + ": translucent objects support max_depth <= 254 (the gather stack holds 255 entries)");
  if (c.dirty_mat_grad || c.mat_grad.size() != c.mats.size()) {
    c.mat_grad.resize(c.mats.size(), nullptr);
    pt_status st = c.d_mat_grad.reserve(std::max<size_t>(c.mats.size(), 1) * sizeof(float*), "gradient table");
    if (st != PT_OK) return st;
    if (!c.mat_grad.empty())
      PT_CHECK_CUDA(cudaMemcpyAsync(c.d_mat_grad.p, c.mat_grad.data(), c.mat_grad.size() * sizeof(float*), cudaMemcpyHostToDevice, c.stream),
                    "gradient table");
    c.dirty_mat_grad = false;
  }
  if (c.dirty_textures) {
    pt_status st = c.d_tex.reserve(std::max<size_t>(c.textures.size(), 1) * sizeof(TexDev), "texture table");
    if (st != PT_OK) return st;
    if (!c.textures.empty())
      PT_CHECK_CUDA(cudaMemcpyAsync(c.d_tex.p, c.textures.data(), c.textures.size() * sizeof(TexDev), cudaMemcpyHostToDevice, c.stream),
                    "texture table");
    c.dirty_textures = false;
  }
  if (c.dirty_materials) {
    PT_CHECK_CUDA(cudaMemcpyAsync(c.d_mats.p, c.mats.data(), c.mats.size() * sizeof(MatDev), cudaMemcpyHostToDevice, c.stream), "material upload");
    PT_CHECK_CUDA(cudaMemcpyAsync(c.d_scat.p, c.scat.data(), c.scat.size() * sizeof(ScatDev), cudaMemcpyHostToDevice, c.stream),
                  "scattering properties upload");
    c.dirty_materials = false;
  }
  DevBuf& geo = c.d_normals_geo;
  if (!geo.p || geo.bytes < (size_t)c.n_tris * sizeof(float4) || c.geo_stale) {
    pt_status st = geo.reserve((size_t)c.n_tris * sizeof(float4), "geometric normals");
    if (st != PT_OK) return st;
    k_geo_normals<<<grid_for(c.n_tris, 256, 8), 256, 0, c.stream>>>(c.view(), geo.as<float4>());
    count_launch();
    c.geo_stale = false;
  }
  return PT_OK;
}

// Camera samples a render of `n_frames` frames of this scene traces (pixels inside the patch).
uint64_t scene_path_samples(const Context& c, uint32_t n_frames)
{
  uint64_t inside_w = (uint64_t)std::min<uint32_t>(c.cam.width, c.cam.patch_origin.x + c.cam.patch_dims.x + 1) -
                      std::min<uint32_t>(c.cam.width, c.cam.patch_origin.x);
  uint64_t inside_h = (uint64_t)std::min<uint32_t>(c.cam.height, c.cam.patch_origin.y + c.cam.patch_dims.y + 1) -
                      std::min<uint32_t>(c.cam.height, c.cam.patch_origin.y);
  return inside_w * inside_h * n_frames;
}

SceneFacts scene_facts(const Context& c)
{
  SceneFacts f;
  f.pixels = c.cam.width * c.cam.height;
  f.n_trans = (uint32_t)c.trans_objs.size();
  f.samples = c.probe_samples;
  f.max_depth = c.integ.max_depth;
  for (const MatDev& m : c.mats)
    if (m.type == MAT_ROUGH_TRANSLUCENT) f.rough = true;
    else if (m.type == MAT_LAMBERTIAN_INTERFACE || m.type == MAT_ROUGH_DIFFUSE) f.layered = true;
    else if ((m.type == MAT_METAL || m.type == MAT_ROUGH_GLASS) && m.model == MULTISCATTERING) f.ms = true;
  return f;
}

PassLayout plan_pass(const std::vector<SceneFacts>& facts, const std::vector<ItemReq>& reqs, uint64_t max_paths, bool dual)
{
  PassLayout L;
  uint32_t max_pixels = 1;
  for (const SceneFacts& f : facts) {
    L.passes = std::max(L.passes, f.max_depth + 2);
    L.layered = L.layered || f.layered;
    L.ms = L.ms || f.ms;
    L.rough = L.rough || f.rough;
    max_pixels = std::max(max_pixels, f.pixels);
    if (f.n_trans) {
      L.sss = true;
      L.g_slots = std::max<uint32_t>(L.g_slots, (uint32_t)f.max_depth + 1);
    }
  }
  if (L.sss) max_paths = std::min<uint64_t>(max_paths, std::max<uint64_t>(max_pixels, (4ull << 30) / ((uint64_t)L.g_slots * 40)));
  if (dual && !L.sss) {
    L.dual = true;
    max_paths = std::max<uint64_t>(1, max_paths / 2);
  }
  uint64_t paths = 0, probes = 0, pix = 0;
  uint32_t sets = 0;
  auto close_chunk = [&]() {
    if (L.chunk_item_begin.size() && L.chunk_item_begin.back() == (uint32_t)L.items.size()) return;
    L.chunk_paths.push_back(paths);
    L.chunk_probes.push_back(probes);
    L.chunk_pixels.push_back(pix);
    L.chunk_sets.push_back(sets);
    L.cap_paths = std::max(L.cap_paths, paths);
    L.cap_probes = std::max(L.cap_probes, probes);
    L.cap_sets = std::max<uint64_t>(L.cap_sets, sets);
    L.chunk_item_begin.push_back((uint32_t)L.items.size());
    paths = probes = pix = 0;
    sets = 0;
  };
  L.chunk_item_begin.push_back(0);
  for (const ItemReq& r : reqs) {
    const SceneFacts& f = facts[r.scene];
    uint32_t done = 0;
    while (done < r.n_frames) {
      uint64_t room = max_paths > paths ? max_paths - paths : 0;
      uint64_t fit = room / f.pixels;
      if ((fit == 0 && paths > 0) || L.items.size() - L.chunk_item_begin.back() >= 65535) {
        close_chunk();
        continue;
      }
      uint32_t take = (uint32_t)std::min<uint64_t>(r.n_frames - done, std::max<uint64_t>(1, fit));
      ItemDev it;
      it.scene = r.scene;
      it.first_frame = r.first_frame + done;
      it.n_frames = take;
      it.pixels = f.pixels;
      it.path_begin = paths;
      it.probe_begin = probes;
      it.pix_begin = pix;
      it.set_begin = sets;
      it.pad = 0;
      L.items.push_back(it);
      paths += (uint64_t)take * f.pixels;
      probes += (uint64_t)take * f.n_trans * f.samples;
      pix += f.pixels;
      sets += take * f.n_trans;
      done += take;
    }
  }
  close_chunk();
  L.chunk_item_begin.pop_back();  // one begin per chunk
  return L;
}

// The scene whose paths alone chunk k of the pass holds, or -1.
static int scene_of_chunk(const PassLayout& L, size_t k)
{
  const uint32_t ib = L.chunk_item_begin[k];
  const uint32_t ie = k + 1 < L.chunk_paths.size() ? L.chunk_item_begin[k + 1] : (uint32_t)L.items.size();
  for (uint32_t i = ib + 1; i < ie; ++i)
    if (L.items[i].scene != L.items[ib].scene) return -1;
  return (int)L.items[ib].scene;
}
static bool all_wide(const std::vector<SceneDev>& scenes)
{
  for (const SceneDev& s : scenes)
    if (!s.nodes4) return false;
  return true;
}
bool chunk_by_pools(const Options& o, const PassLayout& L, uint64_t n, bool multi, bool w4)
{
  return o.pool && w4 && o.extend_mode == 1 && (o.pool == 2 || n <= pool_max_paths(L.sss, L.ms || L.layered || L.rough, multi));
}
bool pass_by_pools(const Options& o, const PassLayout& L, const std::vector<SceneDev>& scenes)
{
  const bool w4 = all_wide(scenes);
  uint64_t all = 0, pools = 0;
  for (size_t k = 0; k < L.chunk_paths.size(); ++k) {
    all += L.chunk_paths[k];
    if (chunk_by_pools(o, L, L.chunk_paths[k], scenes.size() > 1 && scene_of_chunk(L, k) < 0, w4)) pools += L.chunk_paths[k];
  }
  return 2 * pools > all;
}

// Allocates what a pass needs in the engine context E and uploads its scene and item tables (on
// E's stream).  Nothing here may run while E's stream is being captured.
pt_status pass_resources(Context& E, const PassLayout& L, const std::vector<SceneDev>& scenes)
{
  pt_status st = ensure_wavefront(E.wf, L.cap_paths);
  if (st == PT_OK && L.dual) st = ensure_wavefront(E.wf2, L.cap_paths);
  // a small pass's probe paths run beside its camera paths, in a wavefront of their own where memory and the
  // caller's bound on the paths in flight allow
  E.probes_beside = st == PT_OK && L.sss && E.opt.pool && E.opt.overlap && L.cap_probes > 0 && L.cap_probes <= kProbesBesideMax &&
                    L.cap_paths + L.cap_probes <= E.max_paths &&
                    (E.opt.pool == 2 || L.cap_paths <= pool_max_paths(true, L.ms || L.layered || L.rough, scenes.size() > 1)) && ensure_probe_wavefront(E.probe_wf, L.cap_probes) == PT_OK;
  if (st == PT_OK && L.sss) st = ensure_sss(E, E.wf.cap, L.g_slots, L.cap_probes, L.cap_sets);
  if (st == PT_OK) st = E.d_scene_tab.reserve(scenes.size() * sizeof(SceneDev), "scene table");
  if (st == PT_OK) st = E.d_item_tab.reserve(std::max<size_t>(L.items.size(), 1) * sizeof(ItemDev), "item table");
  if (st != PT_OK) return st;
  E.pass_w4 = all_wide(scenes);
  // the overlapped schedule's streams and events (created here, outside any graph capture)
  for (cudaStream_t& sd : E.side)
    if (!sd) PT_CHECK_CUDA(cudaStreamCreateWithFlags(&sd, cudaStreamNonBlocking), "side stream");
  for (cudaEvent_t* ev : {&E.ev_fork, &E.ev_join, &E.ev_shade, &E.ev_shadow})
    if (!*ev) PT_CHECK_CUDA(cudaEventCreateWithFlags(ev, cudaEventDisableTiming), "stream event");
  if (L.dual || E.probes_beside) {
    if (!E.stream2) PT_CHECK_CUDA(cudaStreamCreateWithFlags(&E.stream2, cudaStreamNonBlocking), "second pipeline stream");
    for (cudaEvent_t* ev : {&E.ev_start, &E.ev_end2})
      if (!*ev) PT_CHECK_CUDA(cudaEventCreateWithFlags(ev, cudaEventDisableTiming), "stream event");
  }
  if (L.dual) {
    for (cudaStream_t* sd : {&E.side2[0], &E.side2[1]})
      if (!*sd) PT_CHECK_CUDA(cudaStreamCreateWithFlags(sd, cudaStreamNonBlocking), "second pipeline stream");
    for (cudaEvent_t* ev : {&E.ev2_fork, &E.ev2_join, &E.ev2_shade, &E.ev2_shadow, &E.ev_acc})
      if (!*ev) PT_CHECK_CUDA(cudaEventCreateWithFlags(ev, cudaEventDisableTiming), "stream event");
  }
  PT_CHECK_CUDA(cudaMemcpyAsync(E.d_scene_tab.p, scenes.data(), scenes.size() * sizeof(SceneDev), cudaMemcpyHostToDevice, E.stream), "scene table");
  PT_CHECK_CUDA(cudaMemcpyAsync(E.d_item_tab.p, L.items.data(), L.items.size() * sizeof(ItemDev), cudaMemcpyHostToDevice, E.stream), "item table");
  return PT_OK;
}

// Launches a planned pass on E's stream: per chunk, the probe pass (chunks with translucent objects),
// the camera paths, the deferred gathers and the accumulation.  Only kernel launches and memsets of
// device state: the whole sequence can be captured into a CUDA graph.  multi: the pass spans
// several scenes (the traversal kernels then read each ray's scene from the table; otherwise S0).
pt_status launch_pass(Context& E, const PassLayout& L, const std::vector<SceneDev>& tab, bool multi_pass, bool allow_events, bool adjoint)
{
  // per chunk: a chunk whose paths all render one scene runs the single-scene kernels on that scene
  // (its record as a kernel parameter, no per-ray scene lookup), else the multi-scene kernels
  SceneDev S0 = tab[0];
  bool multi = multi_pass;
  Context& c = E;
  // the device view of one wavefront (dual passes: one per pipeline)
  auto make_w = [&](Wavefront& wf) {
    WfDev v;
    float4* rays = wf.rays.as<float4>();
    float4* state = wf.state.as<float4>();
    v.ray_o = Field2<float4>{rays};
    v.ray_d = Field2<float4>{rays + 1};
    v.thr = Field2<float4>{state};
    v.rad = wf.rad.as<float4>();
    v.rng = Field2<uint4>{reinterpret_cast<uint4*>(state + 1)};
    v.hit = wf.hit.as<float4>();
    v.q_mat = wf.q_mat.as<uint32_t>();
    v.cls_of = wf.cls_of.as<uint8_t>();
    v.bin = wf.bin.as<uint32_t>();
    v.sh_o = wf.sh_o.as<float4>();
    v.sh_d = wf.sh_d.as<float4>();
    v.sh_c = wf.sh_c.as<float4>();
    v.sh_pid = wf.sh_pid.as<uint32_t>();
    v.cnt = wf.counters.as<uint32_t>();
    v.cap = wf.cap;
    v.g_a = L.sss ? wf.g_a.as<float4>() : nullptr;
    v.g_b = L.sss ? wf.g_b.as<float4>() : nullptr;
    v.g_c = L.sss ? wf.g_c.as<float2>() : nullptr;
    v.g_d = L.sss ? wf.g_d.as<float4>() : nullptr;
    v.g_slots = L.sss ? wf.gather_slots : 0;
    v.scenes = c.d_scene_tab.as<SceneDev>();
    v.multi = multi ? 1u : 0u;
    v.scene0 = 0;
    v.path_item = wf.path_item.as<uint16_t>();
    v.adj_a = adjoint ? wf.adj_a.as<float4>() : nullptr;
    v.adj_b = adjoint ? wf.adj_b.as<float4>() : nullptr;
    return v;
  };
  const size_t n_chunks = L.chunk_paths.size();
  const bool prof = c.profile && allow_events;
  // two pipelines: chunk k runs on wavefront k % 2 with that pipeline's streams; the accumulations
  // (each chunk's frames folded into its scenes' running means) stay in chunk order
  const bool dual = L.dual && !adjoint && !prof && n_chunks >= 2 && c.stream2 && c.wf2.cap >= L.cap_paths;
  const WfDev w_of[2] = {make_w(c.wf), dual ? make_w(c.wf2) : make_w(c.wf)};
  Wavefront* const wf_of[2] = {&c.wf, dual ? &c.wf2 : &c.wf};
  WfDev w = w_of[0];
  Wavefront* wf = wf_of[0];
  c.pass_second = dual ? &c.wf2.counters : c.probes_beside ? &c.probe_wf.buf : nullptr;
  Wavefront& wf0 = c.wf;
  SssDev g;
  memset(&g, 0, sizeof(g));
  if (L.sss) {
    g.probes = wf0.probes.as<float4>();
    g.pc_pos = wf0.pc_pos.as<float4>();
    g.pc_wl = wf0.pc_wl.as<float4>();
    g.pc_nrm = wf0.pc_nrm.as<float4>();
    g.pc_tr = wf0.pc_tr.as<float4>();
    g.pc_cnt = wf0.pc_cnt.as<uint32_t>();
  }
  const int grid_trace = sm_count() * 8;
  // the 4-wide BVH when every scene of the pass has one (pass_resources)
  const bool w4 = E.pass_w4;
  // persistent grids: the SM count times the resident blocks of the single- and multi-scene kernels
  int grid_persist_of[2] = {0, 0};
  auto occupancy = [&](auto ext, auto sh, int& grid) -> pt_status {
    int occ_ext = 0, occ_sh = 0;
    PT_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_ext, ext, kTraceBlock, 0), "occupancy");
    PT_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_sh, sh, kTraceBlock, 0), "occupancy");
    grid = sm_count() * std::max(1, std::min(occ_ext, occ_sh));
    return PT_OK;
  };
  pt_status ost;
  if (w4) ost = occupancy(k_extend_persistent<false, true>, k_shadow_persistent<false, false, true>, grid_persist_of[0]);
  else ost = occupancy(k_extend_persistent<false, false>, k_shadow_persistent<false, false, false>, grid_persist_of[0]);
  if (ost == PT_OK && multi_pass) {
    if (w4) ost = occupancy(k_extend_persistent<true, true>, k_shadow_persistent<true, false, true>, grid_persist_of[1]);
    else ost = occupancy(k_extend_persistent<true, false>, k_shadow_persistent<true, false, false>, grid_persist_of[1]);
  }
  if (ost != PT_OK) return ost;
  int grid_persist = grid_persist_of[0];
  const int grid_bin = sm_count() * 8;
  PT_CHECK_CUDA(cudaMemsetAsync(w_of[0].cnt, 0, kCounters * 4, c.stream), "reset counters");
  if (dual) {  // the second pipeline starts after everything queued on the context stream so far
    PT_CHECK_CUDA(cudaEventRecord(c.ev_start, c.stream), "second pipeline start");
    PT_CHECK_CUDA(cudaStreamWaitEvent(c.stream2, c.ev_start, 0), "second pipeline start");
    PT_CHECK_CUDA(cudaMemsetAsync(w_of[1].cnt, 0, kCounters * 4, c.stream2), "reset counters");
  }
  if (c.probes_beside) PT_CHECK_CUDA(cudaMemsetAsync(c.probe_wf.buf.p, 0, kCounters * 4, c.stream), "reset counters");
  c.prof_pairs = 0;
  pt_status st = PT_OK;
  // CUDA events around the launches whose device time the stats report (when profiling is on)
  auto prof_begin = [&](int kind) -> pt_status {
    if (!prof) return PT_OK;
    while (c.prof_events.size() < 2 * (size_t)(c.prof_pairs + 1)) {
      cudaEvent_t ev;
      PT_CHECK_CUDA(cudaEventCreate(&ev), "profiling event");
      c.prof_events.push_back(ev);
    }
    if (c.prof_kind.size() < (size_t)c.prof_pairs + 1) c.prof_kind.resize(c.prof_pairs + 1);
    c.prof_kind[c.prof_pairs] = kind;
    PT_CHECK_CUDA(cudaEventRecord(c.prof_events[2 * c.prof_pairs], c.stream), "profiling event");
    return PT_OK;
  };
  auto prof_end = [&]() -> pt_status {
    if (!prof) return PT_OK;
    PT_CHECK_CUDA(cudaEventRecord(c.prof_events[2 * c.prof_pairs + 1], c.stream), "profiling event");
    ++c.prof_pairs;
    return PT_OK;
  };
  // the current chunk's pipeline: its stream, side streams and events (pipeline 0: the context's)
  cudaStream_t s_main = c.stream;
  cudaEvent_t e_fork = c.ev_fork, e_join = c.ev_join, e_shade = c.ev_shade, e_shadow = c.ev_shadow;
  auto reset_queues = [&]() -> pt_status {
    w.q_in = wf->q_a.as<uint32_t>();
    w.q_out = wf->q_b.as<uint32_t>();
    w.in_slot = CNT_ACTIVE_A;
    w.out_slot = CNT_ACTIVE_B;
    PT_CHECK_CUDA(cudaMemsetAsync(w.cnt, 0, (CNT_FETCH_SH + 1) * 4, s_main), "reset queues");
    return PT_OK;
  };
  // The overlapped schedule (option "overlap", off while profiling so that the extend events time the
  // extend kernel alone).  A bounce's shading kernels work on disjoint paths and only append to the
  // next-ray and shadow-ray queues through atomics, so the smaller classes (miss, light, conductor,
  // dielectric) run on side[0] beside the diffuse, layered and translucent kernels on the context
  // stream.  The shadow rays of bounce b touch only the shadow queue, the path radiance (and, in the
  // adjoint, the adjoint state and gradients); the extend and binning of bounce b + 1 touch neither,
  // so the shadow kernel runs on side[1] beside them, and bounce b + 1's shading, which rewrites the
  // shadow queue and adds to the radiance, waits for it.  Every path's arithmetic is its own, so the
  // images do not depend on the schedule.
  const bool overlap = c.opt.overlap && !prof && c.side[0] && c.side[1] && (!dual || (c.side2[0] && c.side2[1]));
  cudaStream_t s_small = overlap ? c.side[0] : c.stream;
  cudaStream_t s_shadow = overlap ? c.side[1] : c.stream;
  auto wait_on = [&](cudaStream_t waiter, cudaStream_t from, cudaEvent_t ev) -> pt_status {
    PT_CHECK_CUDA(cudaEventRecord(ev, from), "stream fork / join");
    PT_CHECK_CUDA(cudaStreamWaitEvent(waiter, ev, 0), "stream fork / join");
    return PT_OK;
  };
  // a chunk of n paths runs its bounces by path pools
  auto by_pools = [&](uint64_t n) { return !prof && chunk_by_pools(c.opt, L, n, multi, w4); };
  const PoolPrograms programs = L.ms || L.layered || L.rough ? POOL_ALL : L.sss ? POOL_TRANSLUCENT : POOL_BASIC;
  // L.passes = max_depth + 2 bounces: every path has ended by then (each shader stops at max_depth).
  auto bounces = [&](uint64_t n, bool adj_pass) -> pt_status {
    const bool adjoint = adj_pass;
    if (by_pools(n)) {
      if ((st = launch_path_pools(S0, w, n, multi, adjoint, programs, c.opt.refill, s_main)) != PT_OK) return st;
      count_launch();
      ++c.stats.extend_launches;
      return PT_OK;
    }
    for (int b = 0; b < L.passes; ++b) {
      PT_CHECK_CUDA(cudaMemsetAsync(w.cnt + CNT_Q_MISS, 0, (CNT_FETCH_EXT - CNT_Q_MISS + 1) * 4, s_main), "reset queues");
      PT_CHECK_CUDA(cudaMemsetAsync(w.cnt + w.out_slot, 0, 4, s_main), "reset queues");
      if ((st = prof_begin(PROF_EXTEND)) != PT_OK) return st;
      if (c.opt.extend_mode == 1) {
        if (w4) {
          if (multi) k_extend_persistent<true, true><<<grid_persist, kTraceBlock, 0, s_main>>>(S0, w, c.opt.refill);
          else k_extend_persistent<false, true><<<grid_persist, kTraceBlock, 0, s_main>>>(S0, w, c.opt.refill);
        } else {
          if (multi) k_extend_persistent<true, false><<<grid_persist, kTraceBlock, 0, s_main>>>(S0, w, c.opt.refill);
          else k_extend_persistent<false, false><<<grid_persist, kTraceBlock, 0, s_main>>>(S0, w, c.opt.refill);
        }
      } else {
        k_extend<<<grid_trace, kBlock, 0, s_main>>>(w);
      }
      if ((st = prof_end()) != PT_OK) return st;
      if (c.opt.bin_items == 4) launch_binning<4>(w, grid_bin, s_main);
      else if (c.opt.bin_items == 16) launch_binning<16>(w, grid_bin, s_main);
      else launch_binning<8>(w, grid_bin, s_main);
      count_launch(3);
      // the previous bounce's shadow rays are done before this bounce's shading refills their queue
      if (overlap && b > 0 && (st = wait_on(s_main, s_shadow, e_shadow)) != PT_OK) return st;
      PT_CHECK_CUDA(cudaMemsetAsync(w.cnt + CNT_SHADOW, 0, (CNT_FETCH_SH - CNT_SHADOW + 1) * 4, s_main), "reset queues");
      if (overlap && (st = wait_on(s_small, s_main, e_fork)) != PT_OK) return st;
      if (adjoint) {
        k_shade_diffuse<true><<<full_wave(k_shade_diffuse<true>), kBlock, 0, s_main>>>(w);
        k_shade_miss<true><<<full_wave(k_shade_miss<true>), kBlock, 0, s_small>>>(w);
        k_shade_light<true><<<full_wave(k_shade_light<true>), kBlock, 0, s_small>>>(w);
        if (L.ms) {
          launch_shade_ms(w, true, s_small);
        } else {
          k_shade_metal<true, false><<<full_wave(k_shade_metal<true, false>), kBlock, 0, s_small>>>(w);
          k_shade_glass<true, false><<<full_wave(k_shade_glass<true, false>), kBlock, 0, s_small>>>(w);
        }
      } else {
        k_shade_diffuse<false><<<full_wave(k_shade_diffuse<false>), kBlock, 0, s_main>>>(w);
        k_shade_miss<false><<<full_wave(k_shade_miss<false>), kBlock, 0, s_small>>>(w);
        k_shade_light<false><<<full_wave(k_shade_light<false>), kBlock, 0, s_small>>>(w);
        if (L.ms) {
          launch_shade_ms(w, false, s_small);
        } else {
          k_shade_metal<false, false><<<full_wave(k_shade_metal<false, false>), kBlock, 0, s_small>>>(w);
          k_shade_glass<false, false><<<full_wave(k_shade_glass<false, false>), kBlock, 0, s_small>>>(w);
        }
      }
      count_launch(6);
      if (L.layered) {
        launch_shade_layered(w, adjoint, s_main);
        count_launch();
      }
      if (L.sss) {
        launch_shade_translucent(w, adjoint, L.rough, s_main);
        count_launch();
      }
      if (overlap) {
        // join the smaller classes, then fork the shadow rays off the joined stream
        if ((st = wait_on(s_main, s_small, e_join)) != PT_OK) return st;
        if ((st = wait_on(s_shadow, s_main, e_shade)) != PT_OK) return st;
      }
      if (c.opt.extend_mode == 1) {
        if (w4) {
          if (multi && adjoint) k_shadow_persistent<true, true, true><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
          else if (multi) k_shadow_persistent<true, false, true><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
          else if (adjoint) k_shadow_persistent<false, true, true><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
          else k_shadow_persistent<false, false, true><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
        } else {
          if (multi && adjoint) k_shadow_persistent<true, true, false><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
          else if (multi) k_shadow_persistent<true, false, false><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
          else if (adjoint) k_shadow_persistent<false, true, false><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
          else k_shadow_persistent<false, false, false><<<grid_persist, kTraceBlock, 0, s_shadow>>>(S0, w, c.opt.refill);
        }
      } else {
        if (adjoint) k_shadow<true><<<grid_trace, kBlock, 0, s_shadow>>>(w);
        else k_shadow<false><<<grid_trace, kBlock, 0, s_shadow>>>(w);
      }
      count_launch();
      ++c.stats.extend_launches;
      std::swap(w.q_in, w.q_out);
      std::swap(w.in_slot, w.out_slot);
    }
    // the last bounce's shadow rays join the context stream before anything reads the radiance
    if (overlap && (st = wait_on(s_main, s_shadow, e_shadow)) != PT_OK) return st;
    return PT_OK;
  };
  const ItemDev* items = c.d_item_tab.as<ItemDev>();
  for (size_t k = 0; k < n_chunks; ++k) {
    const int pl = dual ? (int)(k & 1) : 0;
    w = w_of[pl];
    wf = wf_of[pl];
    s_main = pl ? c.stream2 : c.stream;
    s_small = overlap ? (pl ? c.side2[0] : c.side[0]) : s_main;
    s_shadow = overlap ? (pl ? c.side2[1] : c.side[1]) : s_main;
    e_fork = pl ? c.ev2_fork : c.ev_fork;
    e_join = pl ? c.ev2_join : c.ev_join;
    e_shade = pl ? c.ev2_shade : c.ev_shade;
    e_shadow = pl ? c.ev2_shadow : c.ev_shadow;
    const uint32_t ib = L.chunk_item_begin[k];
    const uint32_t ie = k + 1 < n_chunks ? L.chunk_item_begin[k + 1] : (uint32_t)L.items.size();
    w.items = items + ib;
    w.n_items = ie - ib;
    multi = multi_pass && scene_of_chunk(L, k) < 0;
    w.multi = multi ? 1u : 0u;
    w.scene0 = multi ? 0u : L.items[ib].scene;
    S0 = tab[w.scene0];
    grid_persist = grid_persist_of[multi ? 1 : 0];
    const uint64_t n_paths = L.chunk_paths[k], n_probes = L.chunk_probes[k];
    // the camera paths do not read the probes (their gathers are evaluated at the end), so where both are
    // small the probe pass runs on a stream and in a wavefront of its own until the gathers
    const bool beside = n_probes && c.probes_beside && n_probes <= c.probe_wf.cap && by_pools(n_paths) && by_pools(n_probes);
    if (beside) {
      WfDev p = w;
      probe_view(c.probe_wf, p);
      p.in_slot = CNT_ACTIVE_A;
      p.out_slot = CNT_ACTIVE_B;
      PT_CHECK_CUDA(cudaEventRecord(c.ev_start, s_main), "probe pass start");
      PT_CHECK_CUDA(cudaStreamWaitEvent(c.stream2, c.ev_start, 0), "probe pass start");
      PT_CHECK_CUDA(cudaMemsetAsync(p.cnt, 0, (CNT_FETCH_SH + 1) * 4, c.stream2), "reset queues");
      k_probe_gen<<<grid_for(n_probes, kBlock, 16), kBlock, 0, c.stream2>>>(p, g, 0, n_probes);
      if ((st = launch_path_pools(S0, p, n_probes, multi, false, programs, c.opt.refill, c.stream2)) != PT_OK) return st;
      k_probe_finish<<<grid_for(n_probes, kBlock, 16), kBlock, 0, c.stream2>>>(p, g, 0, n_probes);
      k_probe_compact<<<L.chunk_sets[k], 256, 0, c.stream2>>>(p, g);
      count_launch(4);
      ++c.stats.extend_launches;
      PT_CHECK_CUDA(cudaEventRecord(c.ev_end2, c.stream2), "probe pass join");
    } else if (n_probes) {
      for (uint64_t j0 = 0; j0 < n_probes; j0 += w.cap) {
        uint64_t nj = std::min<uint64_t>(w.cap, n_probes - j0);
        if ((st = reset_queues()) != PT_OK) return st;
        k_probe_gen<<<grid_for(nj, kBlock, 16), kBlock, 0, s_main>>>(w, g, j0, nj);
        count_launch();
        if ((st = bounces(nj, false)) != PT_OK) return st;
        k_probe_finish<<<grid_for(nj, kBlock, 16), kBlock, 0, s_main>>>(w, g, j0, nj);
        count_launch();
      }
      k_probe_compact<<<L.chunk_sets[k], 256, 0, s_main>>>(w, g);
      count_launch();
    }
    if ((st = reset_queues()) != PT_OK) return st;
    if (adjoint) k_raygen<true><<<grid_for(n_paths, kBlock, 16), kBlock, 0, s_main>>>(w, n_paths);
    else k_raygen<false><<<grid_for(n_paths, kBlock, 16), kBlock, 0, s_main>>>(w, n_paths);
    count_launch();
    if ((st = bounces(n_paths, adjoint)) != PT_OK) return st;
    if (n_probes) {
      if (beside) PT_CHECK_CUDA(cudaStreamWaitEvent(s_main, c.ev_end2, 0), "probe pass join");
      PT_CHECK_CUDA(cudaMemsetAsync(w.cnt + CNT_GATHER, 0, 8, s_main), "reset gather list");
      uint32_t* list = wf->q_a.as<uint32_t>();
      k_gather_collect<<<grid_for(n_paths, kBlock, 16), kBlock, 0, s_main>>>(w, n_paths, list);
      if ((st = prof_begin(PROF_GATHER)) != PT_OK) return st;
      if (adjoint) k_gather<true><<<full_wave(k_gather<true>), kBlock, 0, s_main>>>(w, g, list, 1u);
      else k_gather<false><<<full_wave(k_gather<false>), kBlock, 0, s_main>>>(w, g, list, 1u);
      if ((st = prof_end()) != PT_OK) return st;
      count_launch(2);
    }
    if (!adjoint) {
      // the running means take the chunks' frames in chunk order
      if (dual && k > 0) PT_CHECK_CUDA(cudaStreamWaitEvent(s_main, c.ev_acc, 0), "accumulation order");
      k_accumulate<<<grid_for(L.chunk_pixels[k], kBlock, 16), kBlock, 0, s_main>>>(w, L.chunk_pixels[k]);
      count_launch();
      if (dual) PT_CHECK_CUDA(cudaEventRecord(c.ev_acc, s_main), "accumulation order");
    }
  }
  if (dual) {  // the second pipeline joins the context stream
    PT_CHECK_CUDA(cudaEventRecord(c.ev_end2, c.stream2), "second pipeline join");
    PT_CHECK_CUDA(cudaStreamWaitEvent(c.stream, c.ev_end2, 0), "second pipeline join");
  }
  PT_CHECK_CUDA(cudaGetLastError(), "render launch");
  return PT_OK;
}

}  // namespace pt

using namespace pt;

extern "C" {

pt_status pt_render_frames(pt_ctx* ctx, uint32_t first_frame, uint32_t n_frames)
{
  if (!ctx) return fail(PT_INVALID_ARG, "null context");
  Context& c = ctx->c;
  pt_status st = prepare_scene(c, "pt_render_frames");
  if (st != PT_OK) return st;
  if (n_frames == 0) return PT_OK;
  SceneFacts f = scene_facts(c);
  if (c.differentiable) {
    // keep what the adjoint needs: each path's radiance and the value of each of its gathers
    const uint64_t n = (uint64_t)n_frames * f.pixels;
    const uint32_t slots = f.n_trans ? (uint32_t)f.max_depth + 1 : 0;
    if (n * (1 + slots) * sizeof(float4) > (16ull << 30)) return fail(PT_CAP_EXCEEDED, "pt_render_frames: differentiable state above 16 GiB");
    if ((st = c.d_adj_L.reserve(n * sizeof(float4), "adjoint path radiance")) != PT_OK) return st;
    if (slots && (st = c.d_adj_G.reserve(n * slots * sizeof(float4), "adjoint gather values")) != PT_OK) return st;
    c.adj_first = first_frame;
    c.adj_frames = n_frames;
    c.adj_slots = slots;
    c.adj_valid = true;
  }
  // profiled renders time the kernels of one wavefront (the extend events are on the context stream)
  PassLayout L = plan_pass({f}, {ItemReq{0, first_frame, n_frames}}, c.max_paths, c.opt.dual && !c.differentiable && !c.profile);
  std::vector<SceneDev> scenes{c.view()};
  if ((st = pass_resources(c, L, scenes)) != PT_OK) return st;
  uint64_t launches0 = pt_kernel_launch_count();
  memset(&c.stats, 0, sizeof(c.stats));
  PT_CHECK_CUDA(cudaEventRecord(c.ev0, c.stream), "event");
  if ((st = launch_pass(c, L, scenes, false, true)) != PT_OK) return st;
  PT_CHECK_CUDA(cudaEventRecord(c.ev1, c.stream), "event");
  c.stats.path_samples = scene_path_samples(c, n_frames);
  c.stats.kernel_launches = (uint32_t)(pt_kernel_launch_count() - launches0);
  c.stats_pending = true;
  // the probe buffer of the last chunk holds the last frames of this scene
  c.probe_last_frames = L.items.empty() ? 0 : L.items.back().n_frames;
  c.next_frame = first_frame + n_frames;
  return PT_OK;
}

pt_status pt_render_adjoint(pt_ctx* ctx, uint32_t first_frame, uint32_t n_frames, const float* d_dimage)
{
  if (!ctx || !d_dimage) return fail(PT_INVALID_ARG, "pt_render_adjoint: null argument");
  Context& c = ctx->c;
  if (!c.differentiable || !c.adj_valid) return fail(PT_NOT_READY, "pt_render_adjoint: needs a forward pt_render_frames with the differentiable option on");
  if (first_frame != c.adj_first || n_frames != c.adj_frames)
    return fail(PT_INVALID_ARG, "pt_render_adjoint: frames differ from the last differentiable forward render");
  for (const MatDev& m : c.mats) {
    if (m.type == PT_METALLIC_SHADER && __float_as_int_host(m.tmap.w) >= 0 && m.dist != PT_GGX_DISTRIBUTION)
      return fail(PT_INVALID_ARG, "pt_render_adjoint: roughness gradients are implemented for the GGX distribution");
    if (m.type == PT_ROUGH_TRANSLUCENT_SHADER)
      return fail(PT_INVALID_ARG, "pt_render_adjoint: rough translucent materials are not differentiable");
    if (m.type == PT_TRANSPARENT_SHADER || m.type == PT_LAMBERTIAN_INTERFACE_SHADER || m.type == PT_ROUGH_DIFFUSE_SHADER)
      return fail(PT_INVALID_ARG, "pt_render_adjoint: transparent, lambertian-interface and rough-diffuse materials are not differentiable");
  }
  pt_status st = prepare_scene(c, "pt_render_adjoint");
  if (st != PT_OK) return st;
  SceneFacts f = scene_facts(c);
  PassLayout L = plan_pass({f}, {ItemReq{0, first_frame, n_frames}}, c.max_paths);
  c.adj_dimg = (const float4*)d_dimage;
  c.adj_dscale = 1.0f / (float)((uint64_t)first_frame + n_frames);
  std::vector<SceneDev> scenes{c.view()};
  c.adj_dimg = nullptr;
  c.adj_dscale = 0.0f;
  if ((st = pass_resources(c, L, scenes)) != PT_OK) return st;
  if ((st = c.wf.adj_a.reserve(c.wf.cap * sizeof(float4), "adjoint path state")) != PT_OK) return st;
  if ((st = c.wf.adj_b.reserve(c.wf.cap * sizeof(float4), "adjoint path state")) != PT_OK) return st;
  uint64_t launches0 = pt_kernel_launch_count();
  memset(&c.stats, 0, sizeof(c.stats));
  PT_CHECK_CUDA(cudaEventRecord(c.ev0, c.stream), "event");
  if ((st = launch_pass(c, L, scenes, false, true, true)) != PT_OK) return st;
  PT_CHECK_CUDA(cudaEventRecord(c.ev1, c.stream), "event");
  c.stats.path_samples = scene_path_samples(c, n_frames);
  c.stats.kernel_launches = (uint32_t)(pt_kernel_launch_count() - launches0);
  c.stats_pending = true;
  return PT_OK;
}

pt_status pt_get_probes(pt_ctx* ctx, void* out, uint64_t capacity, uint64_t* n_out)
{
  if (!ctx || !n_out) return fail(PT_INVALID_ARG, "pt_get_probes: null argument");
  Context& c = ctx->c;
  PT_CHECK_CUDA(cudaSetDevice(c.device), "cudaSetDevice");
  const uint64_t per_frame = (uint64_t)c.trans_objs.size() * c.probe_samples;
  if (c.probe_last_frames == 0 || per_frame == 0 || !c.wf.probes.p) {
    *n_out = 0;
    return PT_OK;
  }
  *n_out = per_frame;
  uint64_t n = std::min(capacity, per_frame);
  if (n && !out) return fail(PT_INVALID_ARG, "pt_get_probes: null output buffer");
  const char* src = (const char*)c.wf.probes.p + (size_t)(c.probe_last_frames - 1) * per_frame * 80;
  if (n) PT_CHECK_CUDA(cudaMemcpyAsync(out, src, (size_t)n * 80, cudaMemcpyDeviceToHost, c.stream), "pt_get_probes");
  PT_CHECK_CUDA(cudaStreamSynchronize(c.stream), "pt_get_probes");
  return PT_OK;
}

pt_status pt_get_render_stats(pt_ctx* ctx, pt_render_stats* out)
{
  if (!ctx || !out) return fail(PT_INVALID_ARG, "pt_get_render_stats: null argument");
  Context& c = ctx->c;
  PT_CHECK_CUDA(cudaSetDevice(c.device), "cudaSetDevice");
  PT_CHECK_CUDA(cudaStreamSynchronize(c.stream), "pt_get_render_stats");
  if (c.stats_pending && c.wf.counters.p) {
    uint32_t h[kCounters], h2[kCounters];
    PT_CHECK_CUDA(cudaMemcpy(h, c.wf.counters.p, sizeof(h), cudaMemcpyDeviceToHost), "read counters");
    const bool two = c.pass_second && c.pass_second->p;
    if (two) PT_CHECK_CUDA(cudaMemcpy(h2, c.pass_second->p, sizeof(h2), cudaMemcpyDeviceToHost), "read counters");
    auto rd64 = [&](int slot) {
      unsigned long long v, v2 = 0;
      memcpy(&v, h + slot, 8);
      if (two) memcpy(&v2, h2 + slot, 8);
      return (uint64_t)(v + v2);
    };
    c.stats.segments = rd64(CNT_SEGMENTS_LO);
    c.stats.shadow_rays = rd64(CNT_SHADOW_TOTAL);
    c.stats.capped_walks = rd64(CNT_CAPPED);
    c.stats.clamped_indices = rd64(CNT_CLAMPED);
    c.stats.dipole_gathers = rd64(CNT_GATHERS);
    c.stats.dipole_pairs = rd64(CNT_PAIRS);
    c.stats.gather_overflows = rd64(CNT_ERROR);
    float ms = 0.0f;
    PT_CHECK_CUDA(cudaEventElapsedTime(&ms, c.ev0, c.ev1), "event time");
    c.stats.gpu_ms = ms;
    float ext = 0.0f, gat = 0.0f;
    for (uint32_t k = 0; k < c.prof_pairs; ++k) {
      float e = 0.0f;
      PT_CHECK_CUDA(cudaEventElapsedTime(&e, c.prof_events[2 * k], c.prof_events[2 * k + 1]), "event time");
      (c.prof_kind[k] == PROF_GATHER ? gat : ext) += e;
    }
    c.stats.extend_ms = ext;
    c.stats.gather_ms = gat;
    c.stats_pending = false;
  }
  *out = c.stats;
  return PT_OK;
}

}  // extern "C"
