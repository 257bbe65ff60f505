// Weight-streaming GEMM for few activation rows (decode batches):
//   C[M, N] = A[M, K] * W[N, K]^T (+ epilogue),  bf16 in, fp32 accumulation.
//
// What bounds it: every weight byte is read once from HBM, so the time is N * K * 2 bytes at copy
// bandwidth as long as enough bytes are in flight and an SM takes in little besides weights; for small
// layers the 4 us of launch, first bytes, last sums and stores.  Measured at 1 row, launches replayed
// from a graph, weights beyond L2 (the kernels of gemm_skinny.cu before): 28672 x 4096 40.5 us (50.9;
// 35.9 at 6.55 TB/s), 4096 x 14336 22.4 (25.4; 17.9), 6144 x 4096 12.5 (14.6; 7.7), 4096 x 4096 9.9
// (13.0; 5.1), 5120 x 2048 8.3 (14.2; 3.2).
//
// The operands are swapped: 128 weight rows are the M side of tcgen05.mma and the activation rows
// its N side, rounded up to 16 (not to 128 as where the activations are the M side).  A K block of
// 64 costs 16 KB of weights and 128 bytes per activation row; with one row that is 18 KB, of which
// 16 KB are weights (48 KB, of which 32 KB, in the kernel of 128 x 256 tiles).  K is split over a
// cluster of up to eight CTAs: each streams its part of the weight tile, parks its fp32 partial sums
// in its own shared memory, and after one cluster barrier every CTA adds up the rows it owns out of
// the others' shared memory.  No workspace in global memory, no counters, no second kernel.
//
// Roles (192 threads): warp 0 TMA, warp 1 tcgen05.mma and the owner of tensor memory, warps 2..5
// move the accumulators to shared memory; all six add up and store.  Every wait is bounded; on a
// wait that runs out the CTA still passes both cluster barriers and leaves.
#include "stream.cuh"

namespace b200 {
namespace stream {

constexpr unsigned int kKernelId = 70;
constexpr int kRowBytes = 128;          // bytes of a row in a K block (the swizzle width)
constexpr int kThreads = 192;
constexpr int kWBytes = BW * kRowBytes;
constexpr int kMaxStages = 16;

// as in the other GEMMs of this library
enum Epi : int {
  kNone = 0, kBias = 1, kSiluMul = 2, kFp32 = 4, kRelu2 = 9, kGelu = 10, kGeluMul = 11
};

struct Args {
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;
  int M, N, K;
  int rows;             // activation rows of a tile: a multiple of 16, at most 128
  int row_tiles;
  int splits;           // CTAs of the cluster
  int stages;
  int epi;
  unsigned int* status;
};

__global__ void __launch_bounds__(kThreads)
    gemm_stream_kernel(const __grid_constant__ CUtensorMap tmW,
                       const __grid_constant__ CUtensorMap tmA, const Args p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int stage_bytes = kWBytes + p.rows * kRowBytes;
  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t abort_word;
  volatile uint32_t* abort_flag = &abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = static_cast<int>(blockIdx.x);
  const int row_tile = static_cast<int>(blockIdx.y) % p.row_tiles;
  const int n0 = (static_cast<int>(blockIdx.y) / p.row_tiles) * BW;
  const int m0 = row_tile * p.rows;
  uint32_t cols = 32;
  while (cols < static_cast<uint32_t>(p.rows)) cols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&done_bar, 1);
    abort_word = 0u;
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmA);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  const int total_kb = (p.K + 63) / 64;
  const int kb_lo = static_cast<int>(static_cast<long long>(split) * total_kb / p.splits);
  const int num_kb =
      static_cast<int>(static_cast<long long>(split + 1) * total_kb / p.splits) - kb_lo;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u, p.status, kKernelId, 0x100u + stage,
                       abort_flag))
          break;
        uint8_t* sw = smem + stage * stage_bytes;
        mbar_expect_tx(&full_bar[stage], stage_bytes);
        tma_load_2d(sw, &tmW, &full_bar[stage], (kb_lo + kb) * 64, n0);
        tma_load_2d(sw + kWBytes, &tmA, &full_bar[stage], (kb_lo + kb) * 64, m0);
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc(BW, p.rows, 1, 1);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase, p.status, kKernelId, 0x200u + stage, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + stage * stage_bytes);
        const uint64_t wdesc = make_desc_k_sw128(sw), adesc = make_desc_k_sw128(sw + kWBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16(tmem, wdesc + static_cast<uint64_t>(k * 2), adesc + static_cast<uint64_t>(k * 2),
                   idesc, (kb > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) umma_commit(&done_bar);
    }
  } else {
    // ---------------- accumulators -> shared memory, [activation row][weight row] ----------------
    // every stage has been consumed when done_bar completes, so the partial sums take their place
    const int q = warp & 3;
    const bool ok = mbar_wait(&done_bar, 0u, p.status, kKernelId, 0x300u, abort_flag);
    tc_fence_after();
    if (ok)
      park_sums(tmem, reinterpret_cast<float*>(smem), q, lane, min(p.M - m0, p.rows));
  }
  __syncwarp();
  tc_fence_before();
  if (p.splits > 1) cluster_arrive_wait();
  else __syncthreads();

  // ---------------- sum over the cluster ----------------
  if (abort_word == 0u) {
    const int used = min(p.M - m0, p.rows);
    if (p.epi == kSiluMul || p.epi == kGeluMul) {
      const int col = (n0 >> 1) + 2 * lane;
      sum_rows<true>(smem, split, p.splits, warp, kThreads / 32, lane, used, [&](int r, float4 v) {
        if (col >= (p.N >> 1)) return;
        const uint32_t o = p.epi == kSiluMul
                               ? pack_bf16x2(gated_f<false>(v.x, v.z), gated_f<false>(v.y, v.w))
                               : pack_bf16x2(gated_f<true>(v.x, v.z), gated_f<true>(v.y, v.w));
        *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.C) +
                                     static_cast<long long>(m0 + r) * p.ldc + col) = o;
      });
    } else {
      const int col = n0 + 4 * lane;
      sum_rows<false>(smem, split, p.splits, warp, kThreads / 32, lane, used, [&](int r, float4 v) {
        if (col >= p.N) return;
        const long long at = static_cast<long long>(m0 + r) * p.ldc + col;
        if (p.epi == kFp32) {
          *reinterpret_cast<float4*>(static_cast<float*>(p.C) + at) = v;
          return;
        }
        if (p.epi == kBias) {
          v.x += __bfloat162float(p.bias[col]);
          v.y += __bfloat162float(p.bias[col + 1]);
          v.z += __bfloat162float(p.bias[col + 2]);
          v.w += __bfloat162float(p.bias[col + 3]);
        } else if (p.epi == kRelu2) {
          v = make_float4(relu2_f(v.x), relu2_f(v.y), relu2_f(v.z), relu2_f(v.w));
        } else if (p.epi == kGelu) {
          v = make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w));
        }
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.C) + at) =
            make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
      });
    }
  }
  // nobody leaves while another CTA may still read its partial sums
  if (p.splits > 1) cluster_arrive_wait();
  else __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, cols);
}

struct Plan {
  int rows, row_tiles, splits, stages;
};

static int smem_bytes(int rows, int stages) {
  const int ring = stages * (kWBytes + rows * kRowBytes), sums = rows * BW * 4;
  return (ring > sums ? ring : sums) + 1024;
}

// Up to 128 activation rows make one tile, more make tiles of 128 (a split of K costs 512 bytes per
// row of traffic between the SMs, at about 25 GB/s per SM: it stays below what it saves up to there).
static Plan make_plan(int M, int N, int K, const int* at_once) {
  Plan pl;
  pl.row_tiles = (M + 127) / 128;
  pl.rows = ((M + pl.row_tiles - 1) / pl.row_tiles + 15) / 16 * 16;
  const Split sp = plan_split((N + BW - 1) / BW * pl.row_tiles, (K + 63) / 64, 4, at_once);
  pl.splits = sp.splits;
  const int room = (sp.per_sm == 2 ? kSmemLimit / 2 - 1024 : kSmemLimit) - 1024;
  pl.stages = room / (kWBytes + pl.rows * kRowBytes);
  if (pl.stages > kMaxStages) pl.stages = kMaxStages;
  return pl;
}

}  // namespace stream
}  // namespace b200

// C[M, N] = A[M, K] * W[N, K]^T for M <= 256.  K, N and the pitches are multiples of 8, pointers
// aligned to 16 bytes (epi 2, 11: gate / up rows interleaved in blocks of 32, N a multiple of 64, C is
// [M, N / 2]; epi 4: C is fp32).  -20: not covered.
B200_API int b200_gemm_stream(const void* A, long long lda, const void* W, long long ldw, void* C,
                              long long ldc, int M, int N, int K, const void* bias, int epi,
                              void* stream) {
  using namespace b200;
  using namespace b200::stream;
  if (M <= 0 || N <= 0) return 0;
  const bool gated = epi == kSiluMul || epi == kGeluMul;
  const bool known = gated || epi == kNone || epi == kBias || epi == kFp32 || epi == kRelu2 ||
                     epi == kGelu;
  if (!known || M > 256 || (gated && (N % 64) != 0)) return -20;
  if (K <= 0 || (K % 8) != 0 || (N % 8) != 0 || (lda % 8) != 0 || (ldw % 8) != 0 || (ldc % 8) != 0)
    return -2;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) |
       reinterpret_cast<uintptr_t>(C)) & 15)
    return -3;
  if (epi == kBias && bias == nullptr) return -5;
  static AtOnce table = {};
  const int* at_once = clusters_at_once(table, gemm_stream_kernel, kThreads);
  if (at_once == nullptr) return -20;
  const Plan pl = make_plan(M, N, K, at_once);
  const int bytes = smem_bytes(pl.rows, pl.stages);
  if (pl.stages < 2 || bytes > kSmemLimit) return -20;
  CUtensorMap tmW, tmA;
  int r = encode_tmap_2d(&tmW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, static_cast<uint64_t>(N),
                         static_cast<uint64_t>(K), static_cast<uint64_t>(ldw) * 2, BW, 64,
                         CU_TENSOR_MAP_SWIZZLE_128B);
  if (r != 0) return r < 0 ? -6 : r;
  r = encode_tmap_2d(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, static_cast<uint64_t>(M),
                     static_cast<uint64_t>(K), static_cast<uint64_t>(lda) * 2, pl.rows, 64,
                     CU_TENSOR_MAP_SWIZZLE_128B);
  if (r != 0) return r < 0 ? -6 : r;
  Args a;
  a.C = C;
  a.ldc = ldc;
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.M = M; a.N = N; a.K = K;
  a.rows = pl.rows; a.row_tiles = pl.row_tiles; a.splits = pl.splits; a.stages = pl.stages;
  a.epi = epi;
  a.status = status_ptr();
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg =
      launch_config(pl.splits, (N + BW - 1) / BW * pl.row_tiles, kThreads, bytes, attr,
                    static_cast<cudaStream_t>(stream));
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_stream_kernel, tmW, tmA, a));
}
