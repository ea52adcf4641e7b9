// Path pools: the kernel and its launch, compiled by pt_pool.cu (basic and translucent programs) and
// pt_pool_all.cu (every program).
#pragma once
#include <algorithm>

#include "pt_wavefront.cuh"

namespace pt {

// ------------------------------------------------------------------ path pools
// Every bounce of a pass in one launch.  A block keeps a pool of at most kPool paths, taken from the
// queue of started paths in shares, and repeats until the queue and the pool are empty:
//   take    new paths into the free places of the pool
//   trace   the pool's closest-hit rays and the shadow rays of its last shading, together, by the
//           block's warps with the ray replacement of k_extend_persistent
//   sort    the traced paths by material class (counts and ranks in shared memory)
//   shade   the classes in batches of one warp; continuing paths stay in the pool
// A path's arithmetic is that of the wavefront kernels (the same functions on the same records), and
// the shadow ray of a vertex is added before the path's next vertex is shaded, so the images are the
// wavefront's bit for bit.
// What bounds it: a phase ends with its slowest ray (barrier stalls 5.7 per issue at 262 K paths), while
// issue slots are 46 % busy.  Many small blocks in different phases evict each other's code instead (8 blocks
// of 128 threads take half as long again), and so do inlined draws.  Against the wavefront's launches,
// several contexts at once: a 96 x 64 frame 786 to 239 us, 512 x 512 879 to 567, one frame of a translucent object
// 942 to 345; pool_max_paths has the line to the wavefront.
//
// Threads per block and places of a pool: two blocks of 512 threads per SM (64 registers) and, with all
// vertex programs, one of 1,024, whose warps are all in the same phase: the large programs then share the
// instruction cache (layered scenes with the multiple-scattering model: 18 % less than two of 512).
__host__ __device__ constexpr int pool_threads(int prog) { return prog == POOL_ALL ? 1024 : 512; }
__host__ __device__ constexpr int pool_size(int prog) { return 4 * pool_threads(prog); }
template <int kProg> struct PoolShared {
  static constexpr int kPoolBlock = pool_threads(kProg), kPool = pool_size(kProg);
  uint2 stk[kRing4 * kPoolBlock];
  uint32_t path[2][kPool];   // the pool's paths, and those that continue
  uint32_t shadow[kPool];    // paths with a shadow ray
  uint16_t order[kPool];     // pool entries by class
  uint8_t cls[kPool];
  uint32_t count[kQueues], start[kQueues], batches[kQueues + 1];
  uint32_t n_next, n_shadow, fetch, batch, taken;
};

// Closest hits of pool entries [0, nc) and occlusion of shadow entries [0, ns).
template <bool kMulti, bool kAdj, int kProg>
__device__ __forceinline__ void pool_trace(const SceneDev& S0, const WfDev& w, PoolShared<kProg>& sm, const uint32_t* path, uint32_t nc, uint32_t ns, int refill)
{
  constexpr int kPoolBlock = pool_threads(kProg);
  const uint32_t n = nc + ns;
  TravGeom g = trav_geom(S0);
  const unsigned lane = threadIdx.x & 31;
  // few rays: each warp takes its share of them and no more, since the lanes of a warp take turns between
  // nodes and leaves (a 96 x 64 frame alone: 8 % less)
  constexpr uint32_t kWarpsOfBlock = kPoolBlock / 32;
  const uint32_t lanes = min(32u, (n + kWarpsOfBlock - 1) / kWarpsOfBlock);
  const unsigned mine = lanes >= 32u ? 0xffffffffu : (1u << lanes) - 1u;
  bool has = false, any = false, drained = false;
  uint32_t pid = 0, e = 0;
  float3 o = f3s(0.0f), d = f3s(0.0f);
  float tmin = 0.0f, tmax = 0.0f;
  RayPre4 rp{};
  Hit h;
  h.t = 0.0f; h.u = h.v = 0.0f; h.prim = -1;
  uint2 spill4[kSpill4];
  Stack4 s4;
  stack4_init(s4, sm.stk + threadIdx.x, kPoolBlock, spill4);
  int cur = kDone4;
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, !has) & mine;
    if (!drained && (__popc(idle) >= refill || idle == mine)) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&sm.fetch, (uint32_t)__popc(idle));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base + __popc(idle) >= n) drained = true;
      const uint32_t i = base + __popc(idle & lanemask_lt());
      if (!has && lane < lanes && i < n) {
        any = i >= nc;
        e = any ? i - nc : i;
        pid = any ? sm.shadow[e] : path[e];
        if constexpr (kMulti) g = trav_geom(scene_of(w, pid));
        const float4 o4 = any ? w.sh_o[pid] : w.ray_o[pid], d4 = any ? w.sh_d[pid] : w.ray_d[pid];
        o = ld3(o4);
        d = ld3(d4);
        if constexpr (kMulti) tmin = any ? o4.w : scene_of(w, pid).integ.scene_epsilon;
        else tmin = any ? o4.w : S0.integ.scene_epsilon;
        tmax = any ? d4.w : kDefaultMax;
        rp = ray_pre4(o, d, g.trav_scale);
        h.t = tmax;
        h.u = h.v = 0.0f;
        h.prim = -1;
        stack4_init(s4, sm.stk + threadIdx.x, kPoolBlock, spill4);
        cur = 0;
        has = true;
      }
    }
    if (__ballot_sync(0xffffffffu, has) == 0) break;
    for (;;) {
      // idle lanes have cur == kDone4, so the phase's two ballots also tell how many lanes have finished (a
      // 96 x 64 frame alone: 8 % less; the wavefront's own loops lost 1 % to the same change)
      const bool lp = is_leaf4(cur), np = is_node4(cur);
      const unsigned lmask = __ballot_sync(0xffffffffu, lp), nmask = __ballot_sync(0xffffffffu, np), busy = lmask | nmask;
      if (busy == 0 || (!drained && __popc(mine & ~busy) >= refill)) break;
      if (lmask && (nmask == 0 || __popc(lmask) >= kLeafVsNodeClosest * __popc(nmask))) {
        if (lp) {
          leaf_closest(g, (uint32_t)cur, o, d, tmin, h);
          cur = any && h.prim >= 0 ? kDone4 : stack4_next(s4, h.t, true);
        }
      } else if (np) {
        cur = trav4_node_closest(g, cur, rp, tmin, h, s4);
      }
    }
    if (has && cur == kDone4) {
      const SceneDev& S = kMulti ? scene_of(w, pid) : S0;
      if (any) {
        if (h.prim < 0 && !(S.n_ana && ana_any(S, o, d, tmin, tmax))) shadow_unoccluded<kAdj>(S, w, pid, pid);
      } else {
        if (S.n_ana) ana_closest(S, o, d, tmin, h);
        w.hit[pid] = make_float4(h.t, h.u, h.v, as_float(h.prim));
        const int cls = h.prim < 0 ? QC_MISS : (uint32_t)h.prim >= S.n_tris ? QC_LIGHT : class_of(__ldg(&S.mats[__ldg(&S.tri_info[h.prim].w)].type));
        sm.cls[e] = (uint8_t)cls;
      }
      has = false;
    }
  }
}

// kProg: the vertex programs compiled in (PoolPrograms).
template <bool kMulti, bool kAdj, int kProg>
__global__ void __launch_bounds__(pool_threads(kProg), kProg == POOL_ALL ? 1 : 2) k_path_pool(const __grid_constant__ SceneDev S0, const __grid_constant__ WfDev w, int refill, uint32_t share)
{
  extern __shared__ __align__(16) unsigned char pool_smem[];
  PoolShared<kProg>& sm = *reinterpret_cast<PoolShared<kProg>*>(pool_smem);
  constexpr int kPoolBlock = pool_threads(kProg), kPool = pool_size(kProg);
  const uint32_t n = w.cnt[w.in_slot];
  uint32_t* fetch = w.cnt + CNT_FETCH_EXT;
  const int t = threadIdx.x;
  const uint32_t lane = t & 31;
  uint32_t clamped = 0, overflow = 0, capped_total = 0;
  uint32_t n_path = 0, n_shadow = 0;  // block-uniform
  unsigned long long traced = 0, shadows = 0;
  int side = 0;
  bool more = true;
  for (;;) {
    // take new paths
    if (more && n_path + 32 <= kPool) {
      if (t == 0) sm.taken = atomicAdd(fetch, min(share, (uint32_t)kPool - n_path));
      __syncthreads();
      const uint32_t first = sm.taken, want = min(share, (uint32_t)kPool - n_path);
      const uint32_t got = first < n ? min(want, n - first) : 0u;
      for (uint32_t i = t; i < got; i += kPoolBlock) sm.path[side][n_path + i] = w.q_in[first + i];
      n_path += got;
      more = first + want < n;
    }
    if (n_path + n_shadow == 0) break;
    if (t == 0) {
      sm.fetch = 0;
      sm.n_next = 0;
      sm.batch = 0;
    }
    if (t < kQueues) sm.count[t] = 0;
    __syncthreads();
    traced += n_path;
    shadows += n_shadow;
    pool_trace<kMulti, kAdj, kProg>(S0, w, sm, sm.path[side], n_path, n_shadow, refill);
    __syncthreads();
    // sort the entries by class: ranks by counting, classes from multiples of 32
    uint32_t rank[kPool / kPoolBlock];
#pragma unroll
    for (int j = 0; j < kPool / kPoolBlock; ++j) {
      const uint32_t i = j * kPoolBlock + t;
      const uint32_t c = i < n_path ? sm.cls[i] : 0xffu;
      const unsigned same = __match_any_sync(0xffffffffu, c);
      const uint32_t leader = __ffs(same) - 1;
      uint32_t base = 0;
      if (lane == leader && c < kQueues) base = atomicAdd(&sm.count[c], (uint32_t)__popc(same));
      rank[j] = __shfl_sync(0xffffffffu, base, leader) + __popc(same & lanemask_lt());
    }
    __syncthreads();
    if (t == 0) {
      uint32_t at = 0, b = 0;
      for (int q = 0; q < kQueues; ++q) {
        sm.start[q] = at;
        sm.batches[q] = b;
        at += sm.count[q];
        b += (sm.count[q] + 31u) / 32u;
      }
      sm.batches[kQueues] = b;
      sm.n_shadow = 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPool / kPoolBlock; ++j) {
      const uint32_t i = j * kPoolBlock + t;
      if (i < n_path && sm.cls[i] < kQueues) sm.order[sm.start[sm.cls[i]] + rank[j]] = (uint16_t)i;
    }
    __syncthreads();
    // shade: one warp per batch of 32 entries of a class
    const uint32_t batches = sm.batches[kQueues];
    for (;;) {
      uint32_t b = 0;
      if (lane == 0) b = atomicAdd(&sm.batch, 1u);
      b = __shfl_sync(0xffffffffu, b, 0);
      if (b >= batches) break;
      // the classes of the longest vertices first
      b = batches - 1 - b;
      int q = 0;
      while (sm.batches[q + 1] <= b) ++q;
      const uint32_t k = (b - sm.batches[q]) * 32u + lane;
      const bool in = k < sm.count[q];
      const uint32_t pid = in ? sm.path[side][sm.order[sm.start[q] + k]] : 0u;
      bool cont = false, shadow = false;
      if (in) {
        const SceneDev& S = kMulti ? scene_of(w, pid) : S0;
        NeeRay nee;
        switch (q) {
          case QC_MISS: miss_path<kAdj>(S, w, pid); break;
          case QC_LIGHT: light_path<kAdj>(S, w, pid); break;
          case QC_DIFFUSE: cont = diffuse_path<kAdj>(S, w, pid, nee, shadow, clamped, overflow); break;
          case QC_METAL: cont = metal_path<kAdj, kProg == POOL_ALL>(S, w, pid, capped_total, overflow); break;
          case QC_GLASS: cont = glass_path<kAdj, kProg == POOL_ALL>(S, w, pid, capped_total, overflow); break;
          case QC_TRANS:
            if constexpr (kProg != POOL_BASIC) {
              int capped = 0;
              cont = translucent_path<kAdj, kProg == POOL_ALL>(S, w, pid, overflow, clamped, capped);
              capped_total += capped;
            }
            break;
          default:
            if constexpr (kProg == POOL_ALL) cont = layered_path<kAdj>(S, w, pid, nee, shadow, clamped, overflow, capped_total);
            break;
        }
        if (shadow) put_nee(w, pid, nee);
      }
      const unsigned mc = __ballot_sync(0xffffffffu, cont), ms = __ballot_sync(0xffffffffu, shadow);
      uint32_t bc = 0, bs = 0;
      if (lane == 0) {
        if (mc) bc = atomicAdd(&sm.n_next, (uint32_t)__popc(mc));
        if (ms) bs = atomicAdd(&sm.n_shadow, (uint32_t)__popc(ms));
      }
      bc = __shfl_sync(0xffffffffu, bc, 0);
      bs = __shfl_sync(0xffffffffu, bs, 0);
      if (cont) sm.path[side ^ 1][bc + __popc(mc & lanemask_lt())] = pid;
      if (shadow) sm.shadow[bs + __popc(ms & lanemask_lt())] = pid;
    }
    __syncthreads();
    n_path = sm.n_next;
    n_shadow = sm.n_shadow;
    side ^= 1;
    __syncthreads();
  }
  if (t == 0 && traced) atomicAdd(cnt64(w.cnt, CNT_SEGMENTS_LO), traced);
  if (t == 0 && shadows) atomicAdd(cnt64(w.cnt, CNT_SHADOW_TOTAL), shadows);
  if (clamped) atomicAdd(cnt64(w.cnt, CNT_CLAMPED), (unsigned long long)clamped);
  if (overflow) atomicAdd(cnt64(w.cnt, CNT_ERROR), (unsigned long long)overflow);
  if (capped_total) atomicAdd(cnt64(w.cnt, CNT_CAPPED), (unsigned long long)capped_total);
}

template <int kProg, class K>
static pt_status launch_pool(K kernel, const SceneDev& S0, const WfDev& w, uint64_t n, int refill, cudaStream_t stream)
{
  // the shared memory is above the static limit, which is raised once per kernel, device and thread
  constexpr size_t smem = sizeof(PoolShared<kProg>);
  static thread_local std::vector<std::pair<std::pair<const void*, int>, int>> cache;
  const void* key = reinterpret_cast<const void*>(kernel);
  int dev = 0, wave = 0;
  PT_CHECK_CUDA(cudaGetDevice(&dev), "path pools");
  for (const auto& e : cache)
    if (e.first.first == key && e.first.second == dev) wave = e.second;
  if (!wave) {
    int blocks = 0;
    PT_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "path pools");
    PT_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, pool_threads(kProg), smem), "path pools");
    wave = sm_count() * std::max(1, blocks);
    cache.push_back({{key, dev}, wave});
  }
  // every block takes an equal share of a small pass
  const uint64_t per = (n + wave - 1) / wave;
  const uint32_t share = (uint32_t)std::min<uint64_t>(pool_size(kProg), std::max<uint64_t>(4, (per + 3) / 4 * 4));
  const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(wave, (n + share - 1) / share));
  kernel<<<grid, pool_threads(kProg), smem, stream>>>(S0, w, refill, share);
  PT_CHECK_CUDA(cudaGetLastError(), "path pool launch");
  return PT_OK;
}

// The instance of one program set for a pass of one or many scenes.
template <bool kAdj, int kProg>
static pt_status launch_pool_scenes(const SceneDev& S0, const WfDev& w, uint64_t n, bool multi, int refill, cudaStream_t stream)
{
  return multi ? launch_pool<kProg>(k_path_pool<true, kAdj, kProg>, S0, w, n, refill, stream)
               : launch_pool<kProg>(k_path_pool<false, kAdj, kProg>, S0, w, n, refill, stream);
}

}  // namespace pt
