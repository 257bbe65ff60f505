// What the GEMMs that stream weights past few activation rows share: the split of K over a cluster of
// CTAs, the sum of its partial sums through the shared memory of the cluster, and the plan of a launch.
//
// A CTA holds fp32 partial sums of 128 weight rows as [activation row][weight row] at the start of its
// dynamic shared memory; CTA s of the cluster owns the activation rows s, s + splits, ...
#pragma once

#include "common.cuh"

namespace b200 {
namespace stream {

constexpr int BW = 128;                 // weight rows of a tile
constexpr int kMaxSplits = 8;
constexpr int kSmemLimit = 231424;      // of one CTA, 1 KB of it for the alignment of the ring

__device__ __forceinline__ void cluster_arrive_wait() { cluster_sync(); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local), "r"(rank));
  return out;
}
__device__ __forceinline__ float4 ld_peer4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}
__device__ __forceinline__ float2 ld_peer2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}

// Accumulators of warp quarter q (tensor-memory lanes 32 q .. 32 q + 31 = weight rows) to the partial
// sums in shared memory.
__device__ __forceinline__ void park_sums(uint32_t tmem, float* sums, int q, int lane, int used) {
  float* part = sums + q * 32 + lane;
#pragma unroll 1
  for (int c = 0; c < used; c += 32) {
    uint32_t r[32];
    tmem_ld_32x32(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (c + i < used) part[(c + i) * BW] = __uint_as_float(r[i]);
  }
}

// The rows that CTA `split` owns, four columns (GATED: two gate and two up columns, whose weight rows
// alternate in blocks of 32) a lane, summed in the order of the K slices: store(row, sums).  All peers'
// values of a row are on their way before the first is added.  WHOLE: the sums are 32-bit integers.  Slice s
// is CTA first + s * step of the cluster.
template <bool GATED, bool WHOLE, typename Store>
__device__ __forceinline__ void sum_rows(const void* smem, int split, int splits, int warp, int warps,
                                         int lane, int used, Store store, int first = 0, int step = 1) {
  const int gate = ((2 * lane) >> 5) * 64 + ((2 * lane) & 31);
  const uint32_t own = smem_u32(smem) + (GATED ? gate : 4 * lane) * 4;
  uint32_t peer[kMaxSplits];
#pragma unroll
  for (int s = 0; s < kMaxSplits; ++s)
    peer[s] = s < splits ? (splits > 1 ? peer_addr(own, first + s * step) : own) : 0u;
  for (int r = split + warp * splits; r < used; r += warps * splits) {
    float4 x[kMaxSplits];
#pragma unroll
    for (int s = 0; s < kMaxSplits; ++s) {
      if (s >= splits) continue;
      const uint32_t a = peer[s] + r * (BW * 4);
      if constexpr (GATED) {
        const float2 g = ld_peer2(a), u = ld_peer2(a + 128);
        x[s] = make_float4(g.x, g.y, u.x, u.y);
      } else {
        x[s] = ld_peer4(a);
      }
    }
    float4 v = x[0];
#pragma unroll
    for (int s = 1; s < kMaxSplits; ++s) {
      if (s >= splits) continue;
      if constexpr (WHOLE) {
        v.x = __int_as_float(__float_as_int(v.x) + __float_as_int(x[s].x));
        v.y = __int_as_float(__float_as_int(v.y) + __float_as_int(x[s].y));
        v.z = __int_as_float(__float_as_int(v.z) + __float_as_int(x[s].z));
        v.w = __int_as_float(__float_as_int(v.w) + __float_as_int(x[s].w));
      } else {
        v.x += x[s].x; v.y += x[s].y; v.z += x[s].z; v.w += x[s].w;
      }
    }
    if constexpr (WHOLE)
      v = make_float4(static_cast<float>(__float_as_int(v.x)), static_cast<float>(__float_as_int(v.y)),
                      static_cast<float>(__float_as_int(v.z)), static_cast<float>(__float_as_int(v.w)));
    store(r, v);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
inline cudaLaunchConfig_t launch_config(int splits, int tiles, int threads, int bytes,
                                        cudaLaunchAttribute* attr, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits, tiles);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = static_cast<size_t>(bytes);
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = splits > 1 ? attr : attr + 1;
  cfg.numAttrs = splits > 1 ? 2 : 1;
  return cfg;
}

// Clusters of every size that run at the same time with one CTA per SM (148, 74, 45, 33, 26, 22, 15,
// 15 on a B200: a cluster lies within a group of SMs).  Filled once per device and kernel.
struct AtOnce {
  int n[64][kMaxSplits + 1];
};
template <typename Kernel>
const int* clusters_at_once(AtOnce& table, Kernel kernel, int threads) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  int* t = table.n[dev];
  if (t[1] != 0) return t;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit) !=
      cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  for (int s = kMaxSplits; s >= 1; --s) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = launch_config(s, 512, threads, kSmemLimit, attr, nullptr);
    cfg.numAttrs = 1;                  // the cluster size alone counts here
    int n = 0;
    if (s == 1) n = sm_count();
    else if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    t[s] = n > 0 || s > 1 ? n : 1;
  }
  return t;
}

// CTAs per SM (1 or 2) and K slices for `tiles` tiles.  Tiles beyond the SM count: no split, two CTAs
// per SM, so that the last wave keeps half of the SMs' rings full (28672 x 4096, 1 row: 40.5 us, 43.0
// with one CTA per SM; copy bandwidth 35.9).  Fewer: the split that gives the most SMs something to do,
// one CTA per SM with a ring of 200 KB or two with half of it (6144 x 4096, 48 tiles: two per SM and
// five slices 12.4 us, one and two slices 12.7; 4096 x 4096, 32 tiles: one and four slices 9.8 us, two
// and six 10.1).  Every slice keeps at least `least` of the `blocks` K blocks.
struct Split {
  int per_sm, splits;
};
// Clusters of s at the same time with `per_sm` CTAs per SM: two CTAs of a cluster may share an SM.
inline int at_once_for(const int* at_once, int s, int per_sm) {
  if (per_sm == 1) return at_once[s];
  return (s & 1) ? 2 * at_once[s] : at_once[s / 2];
}
inline Split plan_split(int tiles, int blocks, int least, const int* at_once) {
  const int sms = at_once[1];
  if (tiles > sms) return {2, 1};
  Split best = {1, 1};
  double most = 0.0;
  for (int o = 1; o <= 2; ++o)
    for (int s = 1; s <= kMaxSplits && s * least <= blocks; ++s) {
      if (s > 1 && at_once_for(at_once, s, o) < tiles) continue;
      double use = static_cast<double>(tiles) * s / (o * sms);
      if (o == 2 && s <= 4) use += 1e-6;             // the same use: two CTAs start sooner
      if (use > most) {
        most = use;
        best = {o, s};
      }
    }
  return best;
}

}  // namespace stream
}  // namespace b200
