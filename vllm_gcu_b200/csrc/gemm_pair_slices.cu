// bf16 GEMM on CTA pairs with the weights on the M side, K split over the pairs of a cluster:
//   C[M, N] = A[M, K] * W[N, K]^T (+ epilogue) for a few hundred rows of layers with few weight tiles.
//
// What bounds it: 4096 x 14336 has 16 tiles of 256 weight rows; with 301 rows in two tiles 32 pairs work and 42
// are idle (gemm_pair_rows.cu), smaller row tiles read the weights more often than the SMs can take them in,
// and one weight tile of 256 rows costs a pair 64 us of K blocks.  Here two to four pairs share a tile's K
// blocks.  Each leaves its fp32 sums in its own shared memory, in the place of the ring, and behind one
// cluster barrier every CTA adds up a share of the rows out of the others' (stream.cuh): no workspace, no
// counters, no second kernel.
//
// Off by default (ops/cuda.py, USE_SPLIT_SUMS): partial sums round otherwise than one sum, as exactly, and layers of 16
// bits carry that on.
//
// Measured, launches replayed from a graph, weights beyond L2 (the kernels that run in its place):
// 301 rows, 4096 x 14336 50 -> 36 us, 4096 x 4096 17.7 -> 15.2, 2112 x 7168 25 -> 15.5; 186 rows, 4864 x 14336 50 -> 32;
// 400 rows, 4096 x 14336 53 -> 44.  Not with a second round of clusters (301 rows, 6144 x 4096 19.5 : 28.7) or
// few K blocks a slice (592 rows, 2632 x 1536 9.3 : 13.0).
//
// Roles (320 threads) and barriers of the main loop as in gemm_pair_rows.cu; all warps add up and store.  Every
// wait is bounded; on one that runs out the CTA still passes both cluster barriers and leaves.
#include "pair.cuh"
#include "stream.cuh"

namespace b200 {
namespace pair_slices {

using namespace b200::pair;

constexpr unsigned int kKernelId = 73;
constexpr int kThreads = 320;
constexpr int kHalfW = 128;              // weight rows of a CTA
constexpr int kMaxRows = 256;            // activation rows of a tile
constexpr int kStages = 6;
constexpr int kWBytes = kHalfW * 128;
constexpr int kStageBytes = kWBytes + kMaxRows / 2 * 128;
constexpr int kSmemBytes = kStages * kStageBytes + 1024;
static_assert(kMaxRows * kHalfW * 4 <= kStages * kStageBytes, "partial sums take the ring's place");

enum Epi : int { kNone = 0, kBias = 1, kSiluMul = 2, kRelu2 = 9, kGelu = 10, kGeluMul = 11 };

struct Args {
  __nv_bfloat16* C;
  long long ldc;
  const __nv_bfloat16* bias;
  int M, N, K;
  int rows, row_tiles;        // rows of a tile (a multiple of 32), tiles
  int slices;                 // pairs of a cluster
  int epi;
  unsigned int* status;
};

// Arrives on the barrier at this shared-memory offset in both CTAs of the pair (pair.cuh has the form for
// clusters of one pair).
__device__ __forceinline__ void commit_pair(uint64_t* bar, uint32_t leader) {
  const uint16_t mask = static_cast<uint16_t>(3u << leader);
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(smem_u32(bar)),
      "h"(mask)
      : "memory");
}

__global__ void __launch_bounds__(kThreads, 1)
    gemm_pair_slices_kernel(const __grid_constant__ CUtensorMap tmW,
                            const __grid_constant__ CUtensorMap tmA, const Args p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t full_bar[kStages], empty_bar[kStages], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t abort_word;
  volatile uint32_t* abort_flag = &abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank(), leader = rank & ~1u;
  const int slice = static_cast<int>(rank >> 1), side = static_cast<int>(rank & 1u);
  const int m0 = static_cast<int>(blockIdx.y) % p.row_tiles * p.rows;
  const int used = min(p.M - m0, p.rows);
  const int n0 = static_cast<int>(blockIdx.y) / p.row_tiles * 256 + side * kHalfW;
  const int total_kb = (p.K + 63) / 64;
  const int kb_lo = static_cast<int>(static_cast<long long>(slice) * total_kb / p.slices);
  const int num_kb = static_cast<int>(static_cast<long long>(slice + 1) * total_kb / p.slices) - kb_lo;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 2);                           // one producer per CTA of the pair
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&done_bar, 1);
    abort_word = 0u;
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmA);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // the other CTAs' barriers exist before anything arrives there
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  grid_release();
  // the first weight tiles come into L2 while the kernels in front still run
  if (threadIdx.x == 0)
    for (int kb = 0; n0 < p.N && kb < num_kb && kb < kStages; ++kb) tma_prefetch_2d(&tmW, (kb_lo + kb) * 64, n0);
  __syncwarp();
  grid_wait();

  if (warp == 0) {
    if (elect_one()) {
      const int half = p.rows / 2;
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u, p.status, kKernelId, 0x100u + stage, abort_flag)) break;
        uint8_t* sw = smem + stage * kStageBytes;
        const uint32_t full = map_to_cta(&full_bar[stage], leader);
        mbar_expect_tx_remote(full, kWBytes + half * 128);
        tma_load_2d_pair(sw, &tmW, full, (kb_lo + kb) * 64, n0);
        tma_load_2d_pair(sw + kWBytes, &tmA, full, (kb_lo + kb) * 64, m0 + side * half);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (side == 0 && elect_one()) {
      const uint32_t idesc = make_idesc(256, p.rows, 1, 1);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase, p.status, kKernelId, 0x200u + stage, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + stage * kStageBytes);
        const uint64_t wdesc = make_desc_k_sw128(sw), adesc = make_desc_k_sw128(sw + kWBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16_pair(tmem, wdesc + static_cast<uint64_t>(k * 2), adesc + static_cast<uint64_t>(k * 2), idesc,
                        (kb | k) != 0 ? 1u : 0u);
        commit_pair(&empty_bar[stage], leader);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) commit_pair(&done_bar, leader);
    }
  } else {
    // ---------------- sums -> shared memory, [activation row][weight row] ----------------
    const int q = warp & 3, set = (warp - 2) >> 2;       // two sets of warps take 32 rows in turn
    if (mbar_wait_warp(&done_bar, 0u, p.status, kKernelId, 0x300u, abort_flag)) {
      tc_fence_after();
      float* part = reinterpret_cast<float*>(smem) + q * 32 + lane;
      for (int c = set * 32; c < used; c += 64) {
        uint32_t r[32];
        tmem_ld_32x32(tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(c), r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (c + i < used) part[(c + i) * kHalfW] = __uint_as_float(r[i]);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();

  // ---------------- sum over the slices: the CTAs of this side ----------------
  if (abort_word == 0u) {
    const int warps = kThreads / 32;
    if (p.epi == kSiluMul || p.epi == kGeluMul) {
      const int col = (n0 >> 1) + 2 * lane;
      stream::sum_rows<true, false>(smem, slice, p.slices, warp, warps, lane, used, [&](int r, float4 v) {
        if (col >= (p.N >> 1)) return;
        *reinterpret_cast<uint32_t*>(p.C + static_cast<long long>(m0 + r) * p.ldc + col) =
            p.epi == kSiluMul ? pack_bf16x2(gated_f<false>(v.x, v.z), gated_f<false>(v.y, v.w))
                              : pack_bf16x2(gated_f<true>(v.x, v.z), gated_f<true>(v.y, v.w));
      }, side, 2);
    } else {
      const int col = n0 + 4 * lane;
      float4 bias = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (p.epi == kBias && col < p.N)
        bias = make_float4(__bfloat162float(p.bias[col]), __bfloat162float(p.bias[col + 1]),
                           __bfloat162float(p.bias[col + 2]), __bfloat162float(p.bias[col + 3]));
      stream::sum_rows<false, false>(smem, slice, p.slices, warp, warps, lane, used, [&](int r, float4 v) {
        if (col >= p.N) return;
        if (p.epi == kRelu2) v = make_float4(relu2_f(v.x), relu2_f(v.y), relu2_f(v.z), relu2_f(v.w));
        else if (p.epi == kGelu) v = make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w));
        *reinterpret_cast<uint2*>(p.C + static_cast<long long>(m0 + r) * p.ldc + col) =
            make_uint2(pack_bf16x2(v.x + bias.x, v.y + bias.y), pack_bf16x2(v.z + bias.z, v.w + bias.w));
      }, side, 2);
    }
  }
  // nobody leaves while another CTA may still read its partial sums
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

static cudaLaunchConfig_t config(int slices, int units, cudaLaunchAttribute* attr, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * slices, units);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * slices;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

// Clusters of `slices` pairs that run at the same time (33, 22 and 15 of two, three and four on a B200)
static int clusters_at_once(int slices) {
  static int table[64][5] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int& n = table[dev][slices];
  if (n == 0) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = config(slices, 512, attr, nullptr);
    cfg.numAttrs = 1;
    cudaError_t e =
        cudaFuncSetAttribute(gemm_pair_slices_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    int at_once = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&at_once, gemm_pair_slices_kernel, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    n = e == cudaSuccess && at_once > 0 ? at_once : -1;
  }
  return n > 0 ? n : 0;
}

}  // namespace pair_slices
}  // namespace b200

// Clusters of `slices` (2 .. 4) pairs that run at the same time, 0 where the device takes none.
B200_API int b200_gemm_pair_slices_at_once(int slices) {
  return slices < 2 || slices > 4 ? 0 : b200::pair_slices::clusters_at_once(slices);
}

// As b200_gemm_pair_rows, with the K blocks of a tile shared by `slices` (2 .. 4) pairs.  -20: not covered.
B200_API int b200_gemm_pair_slices(const void* A, long long lda, const void* W, long long ldw, void* C,
                                   long long ldc, int M, int N, int K, const void* bias, int epi, int rows,
                                   int slices, void* stream) {
  using namespace b200;
  using namespace b200::pair_slices;
  if (M <= 0 || N <= 0) return 0;
  const bool gated = epi == kSiluMul || epi == kGeluMul;
  if (!(gated || epi == kNone || epi == kBias || epi == kRelu2 || epi == kGelu) || (gated && (N % 64) != 0) ||
      rows <= 0 || rows > kMaxRows || (rows % 32) != 0 || slices < 2 || slices > 4)
    return -20;
  if (K <= 0 || (K % 8) != 0 || (N % 8) != 0 || (lda % 8) != 0 || (ldw % 8) != 0 || (ldc % 8) != 0) return -2;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(C)) & 15)
    return -3;
  if (epi == kBias && bias == nullptr) return -5;
  if ((K + 63) / 64 < slices || clusters_at_once(slices) == 0) return -20;
  Args a = {};
  a.row_tiles = (M + rows - 1) / rows;
  a.rows = ((M + a.row_tiles - 1) / a.row_tiles + 31) / 32 * 32;
  a.row_tiles = (M + a.rows - 1) / a.rows;
  CUtensorMap tmW, tmA;
  int r = encode_tmap_2d(&tmW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, N, static_cast<uint64_t>(K),
                         static_cast<uint64_t>(ldw) * 2, kHalfW, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r == 0)
    r = encode_tmap_2d(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, M, static_cast<uint64_t>(K),
                       static_cast<uint64_t>(lda) * 2, a.rows / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r != 0) return r < 0 ? -6 : r;
  a.C = static_cast<__nv_bfloat16*>(C);
  a.ldc = ldc;
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.M = M; a.N = N; a.K = K;
  a.epi = epi;
  a.slices = slices;
  a.status = status_ptr();
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg =
      config(slices, (N + 255) / 256 * a.row_tiles, attr, static_cast<cudaStream_t>(stream));
  return launch_code(cudaLaunchKernelEx(&cfg, gemm_pair_slices_kernel, tmW, tmA, a));
}

B200_API int b200_gemm_pair_rows(const void* A, long long lda, const void* W, long long ldw, void* C, long long ldc,
                                 int M, int N, int K, const void* bias, int epi, int rows, void* stream);

// The first `head` weight rows (a multiple of 256) in full rounds of gemm_pair_rows.cu in tiles of `rows`, the others
// here in tiles of `tail_rows`: a last round that a few pairs would work through alone is shared by more.  301 x 28672
// x 4096 (224 tiles over 74 pairs) 74.5 -> 71.1 us, 200 x 20480 x 4096 48.7 -> 43.5, 310 x 9728 x 4096 35.2 -> 30.8, 600 x
// 6400 x 4096 39.3 -> 32.8.  (Starting it without a wait for the kernel in front gave another 0.3 us and was left out.)
B200_API int b200_gemm_pair_rows_tail(const void* A, long long lda, const void* W, long long ldw, void* C,
                                      long long ldc, int M, int N, int K, const void* bias, int epi, int rows,
                                      int head, int tail_rows, int slices, void* stream) {
  using namespace b200;
  using namespace b200::pair_slices;
  if (M <= 0 || N <= 0) return 0;
  if (head <= 0 || head >= N || (head % 256) != 0 || slices < 2 || slices > 4 || tail_rows <= 0 ||
      tail_rows > kMaxRows || (tail_rows % 32) != 0 || (K + 63) / 64 < slices || clusters_at_once(slices) == 0)
    return -20;
  // (the tail's own refusals, before the head runs)
  const bool gated = epi == kSiluMul || epi == kGeluMul;
  if ((N % (gated ? 64 : 8)) != 0) return -20;
  const int rc = b200_gemm_pair_rows(A, lda, W, ldw, C, ldc, M, head, K, bias, epi, rows, stream);
  if (rc != 0) return rc;
  return b200_gemm_pair_slices(A, lda, static_cast<const __nv_bfloat16*>(W) + head * ldw, ldw,
                               static_cast<__nv_bfloat16*>(C) + (gated ? head / 2 : head), ldc, M, N - head, K,
                               bias == nullptr ? nullptr : static_cast<const __nv_bfloat16*>(bias) + head, epi,
                               tail_rows, slices, stream);
}
