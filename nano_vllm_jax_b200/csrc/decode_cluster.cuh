// Pieces shared by the decode kernels that run on thread-block clusters: the cluster's ranks and distributed shared memory,
// 16-byte copies, the warp-level tensor-core tiles, and the choice and launch of a cluster size.
#pragma once

#include <type_traits>

#include "cluster.cuh"
#include "decode_parts.cuh"

namespace nvj {

constexpr int kClMaxCluster = 16;
constexpr int kClMaxRows = 65535;  // a row per grid z

__device__ __forceinline__ void cl_copy16_or_zero(uint32_t dst, const char* src, uint32_t size) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(size) : "memory");
}
__device__ __forceinline__ void cm_ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cm_ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t cm_transpose(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
template <typename T>
__device__ __forceinline__ void cm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __half>::value)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two weights as a 16-bit pair (x low): rounded, or with `rest` what the rounding left over.
template <typename T>
__device__ __forceinline__ uint32_t cm_pack(float x, float y, bool rest) {
  if constexpr (std::is_same<T, __half>::value) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    return rest ? *reinterpret_cast<const uint32_t*>(&l) : *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - __low2float(h), y - __high2float(h));
    return rest ? *reinterpret_cast<const uint32_t*>(&l) : *reinterpret_cast<const uint32_t*>(&h);
  }
}

// Clusters of `cluster` CTAs: one per row and KV head (`heads` of them), or per row where they span the heads (cluster.y).
template <class... Params, class... Args>
inline int launch_clusters(void (*kernel)(Params...), PerDeviceFlags& opted_in, const DecodeParams& p, dim3 cluster, int heads, int threads,
                           int smem, cudaStream_t stream, const Args&... args) {
  if (!once_per_device(opted_in, [&](int) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
               cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
      }))
    return NVJ_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster.x, heads, p.batch);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster.x;
  attr[0].val.clusterDim.y = cluster.y;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...) == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

// CTAs per cluster for `groups` clusters of rows of up to `blocks` blocks, when a CTA walks `walkers` blocks at a time: as many
// as fit the SMs (`per_sm` hundredths of a CTA per SM), at most one per `walkers` blocks of the longest row; and, in batches
// of many CTAs, doubled (up to `grown`) until no walker has more than 12 blocks, so that the last CTAs to finish are short ones.
// Clusters of more than 8 (no longer portable, and placed one by one) only up to 2.2 CTAs per SM.  Any size will do, not only
// powers of two: with those, 28 rows of 128 - 2048 keys took 21.1 us (18.3 with 7 CTAs), 32 rows 21.1 (19.7 with 6), 64 rows of
// 64 - 512 14.9 (13.9 with 3), 64 of 512 - 4096 57.7 (56.2 with 6).  (Measured at 4 - 160 rows: within 3% of each one's best.)
inline int cluster_size(long long groups, int blocks, int sms, int walkers, int per_sm, int grown, int most) {
  auto fitting = [&](int hundredths) { return (int)((long long)hundredths * sms / (100 * groups)); };
  int c = fitting(per_sm);
  if (c > 8) {
    c = fitting(per_sm < 220 ? per_sm : 220);
    c = c > 8 ? c : 8;
  }
  c = c > 1 ? c : 1;
  while (c < grown && blocks > 12 * c * walkers) c = c < 4 ? 2 * c : grown;
  const int useful = (blocks + walkers - 1) / walkers;
  c = c < useful ? c : useful > 1 ? useful : 1;
  c = c < most ? c : most;
  return c;
}
// CTAs of 64 KiB go three to an SM; 2.75, because clusters do not pack every SM.
constexpr int kCmPerSm = 275;

}  // namespace nvj
