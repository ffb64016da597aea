// Thread-block clusters: ranks, the cluster's barrier, loads and stores in another CTA's shared memory.
#pragma once

#include "nvj_common.cuh"

namespace nvj {

__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The barrier in two halves, by whole warps.  The arrival is a release: what the thread has read and written in front of it comes before
// what the others do behind their wait.
__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_sync() {
  cl_arrive();
  cl_wait();
}
// The barrier that keeps a CTA until the others have read its shared memory; nothing that was stored in front is read behind it.  `odd`
// has to depend on every value that the thread has loaded from the others (cl_not_finite of the results is enough): which of the two
// arrivals a warp takes is then only known once all of its loads have returned, so that none can be left for when the CTA it reads
// from has gone, although the usual arrival, a relaxed one, orders nothing by itself.  A release in its place waits for the output's
// stores, or in front of them for its fence: 0.3 us per launch either way, also when one warp releases for the whole CTA (six layers of 48 rows
// 153.6 : 155.6 us, 512 tokens behind 1024 19.1 : 19.5, f32, 8 rows of 64 - 512 keys 7.7 : 8.1).
__device__ __forceinline__ void cl_sync_read(bool odd) {
  if (__any_sync(0xffffffffu, odd)) cl_arrive();
  else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  cl_wait();
}
__device__ __forceinline__ bool cl_not_finite(float4 v) {
  const float s = (v.x + v.y) + (v.z + v.w);
  return !(s - s == 0.f);
}
// Address of this CTA's shared-memory location in CTA `rank` of the cluster, and loads from there.
__device__ __forceinline__ uint32_t cl_map(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 cl_ld4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 cl_ld2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void cl_st2(uint32_t a, float x, int y) {
  asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(__float_as_uint(x)), "r"(y) : "memory");
}

}  // namespace nvj
