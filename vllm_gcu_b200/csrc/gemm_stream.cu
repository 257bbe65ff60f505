// Weight-streaming GEMM for few activation rows (decode batches):
//   C[M, N] = A[M, K] * W[N, K]^T (+ epilogue),  bf16 in, fp32 accumulation;
//   the same of fp8 (e4m3, fp32 accumulation) or int8 (int32) rows with a scale per activation row and
//   per weight row;
//   the experts of a mixture, bf16: rows sorted by expert in tiles of 128, few of them in use.
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
// Experts: a CTA takes 128 weight rows of one expert and the rows in use of one row tile, rounded up to
// 16 (the tile's padding is neither loaded nor multiplied nor stored); no split of K, up to three CTAs
// per SM, so that the start of one runs under the stream of another.  64 tokens, 8 of 128 experts, w13
// 1536 x 2048: 210 -> 115 us, w2 2048 x 768: 107 -> 61 (118 and 59 at copy bandwidth) against tiles of
// 128 x 256 of which a token row is one in thirty.
//
// 8-bit rows: 64 x 28672 x 4096 32.7 -> 26.5 us, 64 x 4096 x 14336 31.3 -> 16.0, 1 x 4096 x 14336
// 39.6 -> 14.9 (9.0 at copy bandwidth) against the persistent tiles of 128 x 128 in gemm_q8.cu.
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
constexpr int kGroupRows = 128;         // rows of a tile of the experts' sorted rows

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
  const float *a_scale, *w_scale;       // 8-bit operands: [M], [N]
  // experts
  const int* expert_ids;                // [M / 128], negative: nothing to do
  const int* num_rows;                  // device scalar: sorted rows in use (a multiple of 128)
  const int* sorted_ids;                // [M], entries from `pairs` on are padding, behind the others
  const float* row_scale;               // optional [M]
  int pairs;
  int ring_bytes;
};

enum Op : int { kBf16 = 0, kFp8 = 1, kInt8 = 2 };

template <int OP>
__device__ __forceinline__ void mma(uint32_t d, uint64_t w, uint64_t x, uint32_t idesc, uint32_t acc) {
  if constexpr (OP == kBf16) umma_f16(d, w, x, idesc, acc);
  else if constexpr (OP == kFp8) umma_f8(d, w, x, idesc, acc);
  else umma_i8(d, w, x, idesc, acc);
}

template <int OP, bool GROUPED>
__global__ void __launch_bounds__(kThreads)
    gemm_stream_kernel(const __grid_constant__ CUtensorMap tmW,
                       const __grid_constant__ CUtensorMap tmA, const Args p) {
  constexpr int kCols = OP == kBf16 ? 64 : 128;        // columns of a K block
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // activation rows [m0, m0 + used) times weight rows [n0, n0 + 128) of a matrix from row w0 on
  int rows, used, m0, n0, w0, split, stages;
  if constexpr (GROUPED) {
    grid_wait();
    m0 = static_cast<int>(blockIdx.y) * kGroupRows;
    if (m0 >= *p.num_rows) return;
    const int expert = p.expert_ids[blockIdx.y];
    const int4 ids = reinterpret_cast<const int4*>(p.sorted_ids + m0)[lane];
    used = static_cast<int>(__reduce_add_sync(
        0xffffffffu, static_cast<unsigned>((ids.x < p.pairs) + (ids.y < p.pairs) +
                                           (ids.z < p.pairs) + (ids.w < p.pairs))));
    if (expert < 0 || used == 0) return;
    n0 = static_cast<int>(blockIdx.x) * BW;
    w0 = expert * p.N;
    rows = (used + 15) & ~15;
    stages = min(p.ring_bytes / (kWBytes + rows * kRowBytes), kMaxStages);
    split = 0;
  } else {
    rows = p.rows;
    m0 = static_cast<int>(blockIdx.y) % p.row_tiles * rows;
    n0 = static_cast<int>(blockIdx.y) / p.row_tiles * BW;
    used = min(p.M - m0, rows);
    w0 = 0;
    stages = p.stages;
    split = static_cast<int>(blockIdx.x);
  }
  const int splits = GROUPED ? 1 : p.splits;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int stage_bytes = kWBytes + rows * kRowBytes;
  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t abort_word;
  volatile uint32_t* abort_flag = &abort_word;
  uint32_t cols = 32;
  while (cols < static_cast<uint32_t>(rows)) cols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
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
  grid_release();

  const int total_kb = (p.K + kCols - 1) / kCols;
  const int kb_lo = static_cast<int>(static_cast<long long>(split) * total_kb / splits);
  const int num_kb =
      static_cast<int>(static_cast<long long>(split + 1) * total_kb / splits) - kb_lo;

  if constexpr (!GROUPED) {
    // The first weight tiles come into L2 while the kernels in front still run (not into shared memory:
    // nothing says that they do not write them)
    if (threadIdx.x == 0)
      for (int kb = 0; kb < num_kb && kb < stages; ++kb)
        tma_prefetch_2d(&tmW, (kb_lo + kb) * kCols, n0);
    __syncwarp();
    grid_wait();
  }

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
        tma_load_2d(sw, &tmW, &full_bar[stage], (kb_lo + kb) * kCols, w0 + n0);
        if constexpr (GROUPED) {
          for (int r = 0; r < rows; r += 16)
            tma_load_2d(sw + kWBytes + r * kRowBytes, &tmA, &full_bar[stage], kb * kCols, m0 + r);
        } else {
          tma_load_2d(sw + kWBytes, &tmA, &full_bar[stage], (kb_lo + kb) * kCols, m0);
        }
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = OP == kBf16   ? make_idesc(BW, rows, 1, 1)
                             : OP == kInt8 ? make_idesc(BW, rows, 1, 1, 2)
                                           : make_idesc(BW, rows, 0, 0, 1);
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
          mma<OP>(tmem, wdesc + static_cast<uint64_t>(k * 2), adesc + static_cast<uint64_t>(k * 2),
                  idesc, (kb > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        if (++stage == stages) {
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
    const bool ok = mbar_wait_warp(&done_bar, 0u, p.status, kKernelId, 0x300u, abort_flag);
    tc_fence_after();
    if (ok)
      park_sums(tmem, reinterpret_cast<float*>(smem), q, lane, used);
  }
  tc_fence_before();
  if (splits > 1) cluster_arrive_wait();
  else __syncthreads();

  // ---------------- sum over the cluster ----------------
  if (abort_word == 0u) {
    if (OP == kBf16 && (p.epi == kSiluMul || p.epi == kGeluMul)) {
      const int col = (n0 >> 1) + 2 * lane;
      sum_rows<true, false>(smem, split, splits, warp, kThreads / 32, lane, used, [&](int r, float4 v) {
        if (col >= (p.N >> 1)) return;
        const uint32_t o = p.epi == kSiluMul
                               ? pack_bf16x2(gated_f<false>(v.x, v.z), gated_f<false>(v.y, v.w))
                               : pack_bf16x2(gated_f<true>(v.x, v.z), gated_f<true>(v.y, v.w));
        *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.C) +
                                     static_cast<long long>(m0 + r) * p.ldc + col) = o;
      });
    } else {
      const int col = n0 + 4 * lane;
      float4 ws = make_float4(1.f, 1.f, 1.f, 1.f);
      if (OP != kBf16 && col < p.N)
        ws = make_float4(p.w_scale[col], p.w_scale[col + 1], p.w_scale[col + 2], p.w_scale[col + 3]);
      sum_rows<false, OP == kInt8>(
          smem, split, splits, warp, kThreads / 32, lane, used, [&](int r, float4 v) {
            if (col >= p.N) return;
            const long long at = static_cast<long long>(m0 + r) * p.ldc + col;
            if constexpr (OP != kBf16) {
              const float s = p.a_scale[m0 + r];
              v = make_float4(v.x * s * ws.x, v.y * s * ws.y, v.z * s * ws.z, v.w * s * ws.w);
            }
            if constexpr (GROUPED) {
              if (p.row_scale != nullptr) {
                const float s = p.row_scale[m0 + r];
                v = make_float4(v.x * s, v.y * s, v.z * s, v.w * s);
              }
            }
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
  if (splits > 1) cluster_arrive_wait();
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
// Smaller ones where K is so short that it leaves no room for a split and SMs for more tiles: moving out
// the sums is most of a tile's time then.  us with one tile of rows : as here (the kernels that went
// before), 128 x 512 x 512 of 8 bits 10.9 : 4.0 (10.0), 256 x 1152 x 896 11.5 : 5.5 (11.1), 32 x 1024 x 128
// of bf16 3.9 : 3.2 (3.5).  With a longer K it does not pay: 17 x 896 x 4864 5.3 : 6.6.
static Plan make_plan(int M, int N, int blocks, const int* at_once) {
  const int tiles = (N + BW - 1) / BW;
  Plan pl;
  Split sp;
  for (pl.row_tiles = (M + 127) / 128;; pl.row_tiles *= 2) {
    const int used = (M + pl.row_tiles - 1) / pl.row_tiles;
    pl.rows = (used + 15) / 16 * 16;
    sp = plan_split(tiles * pl.row_tiles, blocks, 4, at_once);
    const int ctas = tiles * pl.row_tiles * sp.splits;
    if (blocks > 8 || pl.rows == 16 || (used > 24 ? 2 : 4) * ctas > at_once[1]) break;
  }
  pl.row_tiles = (M + pl.rows - 1) / pl.rows;
  pl.splits = sp.splits;
  const int room = (sp.per_sm == 2 ? kSmemLimit / 2 - 1024 : kSmemLimit) - 1024;
  pl.stages = room / (kWBytes + pl.rows * kRowBytes);
  if (pl.stages > kMaxStages) pl.stages = kMaxStages;
  return pl;
}

// Rows of 128 bytes in both tensor maps: bf16 or one-byte elements.
static int make_maps(int op, const void* W, uint64_t w_rows, long long ldw, const void* A,
                     uint64_t a_rows, long long lda, uint64_t K, int a_box, CUtensorMap* tmW,
                     CUtensorMap* tmA) {
  const int size = op == kBf16 ? 2 : 1, cols = kRowBytes / size;
  const CUtensorMapDataType type =
      op == kBf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  int r = encode_tmap_2d(tmW, type, size, W, w_rows, K, static_cast<uint64_t>(ldw) * size, BW, cols,
                         CU_TENSOR_MAP_SWIZZLE_128B);
  if (r == 0)
    r = encode_tmap_2d(tmA, type, size, A, a_rows, K, static_cast<uint64_t>(lda) * size, a_box, cols,
                       CU_TENSOR_MAP_SWIZZLE_128B);
  return r < 0 ? -6 : r;
}

// Dense: p has C, ldc, bias, M, N, K, epi and scales.
template <int OP>
static int launch(const void* A, long long lda, const void* W, long long ldw, Args p,
                  cudaStream_t stream) {
  static AtOnce table = {};
  auto kernel = gemm_stream_kernel<OP, false>;
  const int* at_once = clusters_at_once(table, kernel, kThreads);
  if (at_once == nullptr) return -20;
  const int cols = OP == kBf16 ? 64 : 128;
  const Plan pl = make_plan(p.M, p.N, (p.K + cols - 1) / cols, at_once);
  const int bytes = smem_bytes(pl.rows, pl.stages);
  if (pl.stages < 2 || bytes > kSmemLimit) return -20;
  CUtensorMap tmW, tmA;
  const int r = make_maps(OP, W, p.N, ldw, A, p.M, lda, p.K, pl.rows, &tmW, &tmA);
  if (r != 0) return r;
  p.rows = pl.rows; p.row_tiles = pl.row_tiles; p.splits = pl.splits; p.stages = pl.stages;
  p.status = status_ptr();
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = launch_config(pl.splits, (p.N + BW - 1) / BW * pl.row_tiles, kThreads,
                                               bytes, attr, stream);
  return launch_code(cudaLaunchKernelEx(&cfg, kernel, tmW, tmA, p));
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
  Args a = {};
  a.C = C;
  a.ldc = ldc;
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.M = M; a.N = N; a.K = K;
  a.epi = epi;
  return launch<kBf16>(A, lda, W, ldw, a, static_cast<cudaStream_t>(stream));
}

// The same of one-byte operands: C (bf16) = A * W^T * a_scale[row] * w_scale[column] (+ bias), M <= 256;
// kind 0 fp8 e4m3, 2 int8; K and the pitches of A and W multiples of 16.
B200_API int b200_gemm_stream_q8(const void* A, long long lda, const void* W, long long ldw, void* C,
                                 long long ldc, int M, int N, int K, const float* a_scale,
                                 const float* w_scale, const void* bias, int kind, void* stream) {
  using namespace b200;
  using namespace b200::stream;
  if (M <= 0 || N <= 0) return 0;
  if (M > 256 || (kind != 0 && kind != 2)) return -20;
  if (K <= 0 || (K % 16) != 0 || (lda % 16) != 0 || (ldw % 16) != 0 || (N % 8) != 0 ||
      (ldc % 8) != 0 || a_scale == nullptr || w_scale == nullptr)
    return -2;
  Args a = {};
  a.C = C;
  a.ldc = ldc;
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.a_scale = a_scale;
  a.w_scale = w_scale;
  a.M = M; a.N = N; a.K = K;
  a.epi = bias != nullptr ? kBias : kNone;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return kind == 0 ? launch<kFp8>(A, lda, W, ldw, a, s) : launch<kInt8>(A, lda, W, ldw, a, s);
}

// Experts: A [M_cap, K] rows sorted by expert in tiles of 128, tile t for expert expert_ids[t]; rows whose
// sorted id is `pairs` or more are padding (the last ones of a tile) and are not written.  W [E, N, K];
// epi as b200_gemm_bf16_grouped.  -20: not covered.
B200_API int b200_gemm_stream_grouped(const void* A, long long lda, const void* W, long long ldw,
                                      void* C, long long ldc, int M_cap, int N, int K, int E,
                                      const int* expert_ids, const int* num_rows,
                                      const int* sorted_ids, int pairs, const float* row_scale, int epi,
                                      void* stream) {
  using namespace b200;
  using namespace b200::stream;
  if (M_cap <= 0 || N <= 0 || E <= 0 || pairs <= 0) return 0;
  if ((M_cap % kGroupRows) != 0 || K <= 0 || (K % 8) != 0 || (lda % 8) != 0 || (ldw % 8) != 0 ||
      (ldc % 8) != 0 || expert_ids == nullptr || num_rows == nullptr || sorted_ids == nullptr)
    return -2;
  if ((N % 64) != 0 || (epi != kNone && epi != kSiluMul && epi != kRelu2 && epi != kGelu)) return -20;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) |
       reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(sorted_ids)) & 15)
    return -20;
  CUtensorMap tmW, tmA;
  const int r = make_maps(kBf16, W, static_cast<uint64_t>(E) * N, ldw, A, M_cap, lda, K, 16, &tmW, &tmA);
  if (r != 0) return r;
  Args a = {};
  a.C = C;
  a.ldc = ldc;
  a.M = M_cap; a.N = N; a.K = K;
  a.epi = epi;
  a.status = status_ptr();
  a.expert_ids = expert_ids; a.num_rows = num_rows; a.sorted_ids = sorted_ids; a.pairs = pairs;
  a.row_scale = row_scale;
  // three CTAs per SM while their tiles hold a few rows; two stages of full tiles have to fit
  const int room = (pairs <= 16LL * E ? kSmemLimit / 3 : kSmemLimit / 2) - 1024;
  a.ring_bytes = room - 1024;
  static_assert((kSmemLimit / 3 - 2048) / (kWBytes + kGroupRows * kRowBytes) >= 2 &&
                    kSmemLimit / 3 - 2048 >= kGroupRows * BW * 4, "ring of a full tile");
  auto kernel = gemm_stream_kernel<kBf16, true>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kSmemLimit);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[dev] = true;
  }
  // Every tile in use holds a pair, so there are no more of them than pairs: room for every expert is
  // mostly empty with a few tokens (one token, 8 of 384 experts of 512 x 512: 3072 CTAs that leave at once,
  // 88 us for both products and what is around them, 78 without)
  dim3 grid((N + BW - 1) / BW, pairs < M_cap / kGroupRows ? pairs : M_cap / kGroupRows);
  return launch_overlapped(kernel, grid, dim3(kThreads), static_cast<size_t>(room),
                           static_cast<cudaStream_t>(stream), tmW, tmA, a);
}
