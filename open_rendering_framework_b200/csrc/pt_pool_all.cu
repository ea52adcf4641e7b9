// Path pools with every vertex program, and the wavefront's shading kernels of the large programs
// (layered, translucent, multiple scattering).  These kernels hold several walks, so the draw and the
// walks' large functions are compiled once, out of line (layered scenes with the multiple-scattering model:
// 13 % less than with the draw alone out of line).
#define PT_OUTLINE_TEA
#define PT_OUTLINE_WALK
#include "pt_pool.cuh"

namespace pt {

pt_status launch_path_pools_all(const SceneDev& S0, const WfDev& w, uint64_t n, bool multi, bool adjoint, int refill, cudaStream_t stream)
{
  return adjoint ? launch_pool_scenes<true, POOL_ALL>(S0, w, n, multi, refill, stream)
                 : launch_pool_scenes<false, POOL_ALL>(S0, w, n, multi, refill, stream);
}

// ------------------------------------------------------------------ the wavefront's large shading kernels
template <bool kAdj>
__global__ void __launch_bounds__(kBlock) k_shade_layered(WfDev w)
{
  __shared__ uint32_t sm[kWarps + 1];
  const uint32_t n = w.cnt[CNT_Q_LAYERED];
  const uint32_t* q = w.q_mat + (size_t)QC_LAYERED * w.cap;
  uint32_t clamped = 0, overflow = 0, capped_total = 0;
  for (uint32_t base = blockIdx.x * kBlock; base < n; base += gridDim.x * kBlock) {
    const uint32_t i = base + threadIdx.x;
    bool shadow = false, cont = false;
    uint32_t pid = 0;
    NeeRay nee;
    if (i < n) {
      pid = q[i];
      cont = layered_path<kAdj>(scene_of(w, pid), w, pid, nee, shadow, clamped, overflow, capped_total);
    }
    const uint32_t s_slot = block_slot(shadow, w.cnt + CNT_SHADOW, sm);
    if (shadow) {
      put_nee(w, s_slot, nee);
      w.sh_pid[s_slot] = pid;
    }
    const uint32_t c_slot = block_slot(cont, w.cnt + w.out_slot, sm);
    if (cont) w.q_out[c_slot] = pid;
  }
  if (clamped) atomicAdd(cnt64(w.cnt, CNT_CLAMPED), (unsigned long long)clamped);
  if (overflow) atomicAdd(cnt64(w.cnt, CNT_ERROR), (unsigned long long)overflow);
  if (capped_total) atomicAdd(cnt64(w.cnt, CNT_CAPPED), (unsigned long long)capped_total);
}

// kRough: some translucent material of the pass has a rough boundary (else that code is left out).
template <bool kAdj, bool kRough>
__global__ void __launch_bounds__(kBlock) k_shade_translucent(WfDev w)
{
  __shared__ uint32_t sm[kWarps + 1];
  const uint32_t n = w.cnt[CNT_Q_TRANS];
  const uint32_t* q = w.q_mat + (size_t)QC_TRANS * w.cap;
  uint32_t overflow = 0, clamped = 0;
  int capped = 0;
  for (uint32_t base = blockIdx.x * kBlock; base < n; base += gridDim.x * kBlock) {
    uint32_t i = base + threadIdx.x;
    bool cont = false;
    uint32_t pid = 0;
    if (i < n) {
      pid = q[i];
      cont = translucent_path<kAdj, kRough>(scene_of(w, pid), w, pid, overflow, clamped, capped);
    }
    uint32_t c_slot = block_slot(cont, w.cnt + w.out_slot, sm);
    if (cont) w.q_out[c_slot] = pid;
  }
  if (overflow) atomicAdd(cnt64(w.cnt, CNT_ERROR), (unsigned long long)overflow);
  if (clamped) atomicAdd(cnt64(w.cnt, CNT_CLAMPED), (unsigned long long)clamped);
  if (capped) atomicAdd(cnt64(w.cnt, CNT_CAPPED), (unsigned long long)capped);
}

void launch_shade_layered(const WfDev& w, bool adjoint, cudaStream_t stream)
{
  if (adjoint) k_shade_layered<true><<<full_wave(k_shade_layered<true>), kBlock, 0, stream>>>(w);
  else k_shade_layered<false><<<full_wave(k_shade_layered<false>), kBlock, 0, stream>>>(w);
}
void launch_shade_translucent(const WfDev& w, bool adjoint, bool rough, cudaStream_t stream)
{
  // the adjoint rejects rough boundaries
  if (adjoint) k_shade_translucent<true, false><<<full_wave(k_shade_translucent<true, false>), kBlock, 0, stream>>>(w);
  else if (rough) k_shade_translucent<false, true><<<full_wave(k_shade_translucent<false, true>), kBlock, 0, stream>>>(w);
  else k_shade_translucent<false, false><<<full_wave(k_shade_translucent<false, false>), kBlock, 0, stream>>>(w);
}
void launch_shade_ms(const WfDev& w, bool adjoint, cudaStream_t stream)
{
  if (adjoint) {
    k_shade_metal<true, true><<<full_wave(k_shade_metal<true, true>), kBlock, 0, stream>>>(w);
    k_shade_glass<true, true><<<full_wave(k_shade_glass<true, true>), kBlock, 0, stream>>>(w);
  } else {
    k_shade_metal<false, true><<<full_wave(k_shade_metal<false, true>), kBlock, 0, stream>>>(w);
    k_shade_glass<false, true><<<full_wave(k_shade_glass<false, true>), kBlock, 0, stream>>>(w);
  }
}

}  // namespace pt
