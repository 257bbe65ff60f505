// bf16 GEMM on CTA pairs with the weights on the M side of the tensor cores:
//   C[M, N] = A[M, K] * W[N, K]^T (+ epilogue) for a few hundred activation rows, and for the experts of
// a mixture (rows sorted by expert in tiles of 128).
//
// What bounds it: between decode batches (weight bytes) and prefill (tensor cores) a tile of 256 rows
// wastes what the rows do not fill: 301 rows make two tiles of 256, an expert with 260 rows three of 128.
// With the operands swapped a pair of CTAs holds 256 weight rows (128 each, M = 256 of
// tcgen05.mma.cta_group::2) and the activation rows are its N side, any multiple of 32 up to 256, of which
// each CTA loads one half: 16 KB of weights and at most 16 KB of rows per K block and CTA, the
// intensity of a 256 x 256 tile when they are full.  Accumulators: 256 columns of tensor memory, two
// sets, so that the epilogue of a tile (two neighbouring lanes exchange a number for every two rows, and each stores
// two columns of one) runs under the MMAs of the next.
//
// Persistent pairs.  Dense: the row tiles of a weight tile follow each other, so that the weights come
// from L2 after the first.  Experts: two row tiles of an expert make one (up to 256 rows), its padding is
// loaded up to the next 32 rows and never stored; every CTA lists the tiles from the sorted rows' tables
// when it starts.
//
// Measured, launches replayed from a graph, weights beyond L2 (the kernels it took over from): 301 rows,
// 28672 x 4096 74 us (89; 44 at the tensor cores' rate, 63 the vendor library), 6144 x 4096 20 (28).  With the first
// epilogue: 36864 x 7168 140 (178); 32 experts of 7168 x 2048 with 256 rows each, w13 466 us (633 in row tiles of 128;
// 321 at the tensor cores' rate), w2 254 (466).
// What held short K was that epilogue, 3000 cycles for 32 rows of a gated product (IEEE divisions that wait for
// one another, four warps that meet three times a chunk) beside 512 of a K block's products.  Eight warps,
// no divisions with branches, neighbours' exchange in place of a transposition: 128 experts, 4096 tokens of 8
// (the same in equal shares): w13 1536 x 2048 260 (216) -> 220 (182), w2 2048 x 768 177 (149) -> 125 (106),
// where the weights and rows take 150 and 90 at copy bandwidth.
//
// Roles (320 threads per CTA; eight epilogue warps) and barriers as in gemm_pair.cu.
#include "pair.cuh"

namespace b200 {
namespace pair_rows {

using namespace b200::pair;

constexpr unsigned int kKernelId = 72;
constexpr int kThreads = 320;
constexpr int kHalfW = 128;              // weight rows of a CTA
constexpr int kMaxRows = 256;            // activation rows of a tile
constexpr int kStages = 6;
constexpr int kWBytes = kHalfW * 128;
constexpr int kStageBytes = kWBytes + kMaxRows / 2 * 128;
constexpr int kChunk = 4 * 4096;         // gate and up values between the epilogue warps
constexpr int kOffOut = kStages * kStageBytes;
constexpr int kSmemBytes = kOffOut + kChunk + 1024;
constexpr int kMaxList = 2048;           // row tiles of a grouped launch, in pairs
static_assert(kSmemBytes + 4 * kMaxList + 1024 <= 232448, "exceeds the shared memory of one CTA");

enum Epi : int { kNone = 0, kBias = 1, kSiluMul = 2, kRelu2 = 9, kGelu = 10, kGeluMul = 11 };

struct Args {
  __nv_bfloat16* C;
  long long ldc;
  const __nv_bfloat16* bias;
  int M, N, K;
  int rows, row_tiles;        // dense: rows of a tile (a multiple of 32), tiles
  int epi;
  unsigned int* status;
  // experts
  const int* expert_ids;      // [M / 128]
  const int* num_rows;        // device scalar: sorted rows in use, a multiple of 128
  const int* tile_rows;       // [M / 128]: rows of every tile that are no padding
  const float* row_scale;     // optional [M]
};

struct Unit {
  int m0, used, rows, n0, w0;  // rows [m0, m0 + used) in a tile of `rows`; weight rows w0 + n0 ...
};

template <bool GROUPED>
__device__ __forceinline__ Unit unit_at(const Args& p, const uint32_t* list, int u) {
  Unit x;
  if constexpr (GROUPED) {
    const int w_tiles = (p.N + 255) / 256;
    const uint32_t e = list[u / w_tiles];
    x.m0 = static_cast<int>(e >> 16) * 128;
    x.used = static_cast<int>(e & 0xFFFFu);
    x.rows = (x.used + 31) & ~31;
    x.n0 = u % w_tiles * 256;
    x.w0 = p.expert_ids[e >> 16] * p.N;
  } else {
    x.m0 = u % p.row_tiles * p.rows;
    x.rows = p.rows;
    x.used = min(p.M - x.m0, p.rows);
    x.n0 = u / p.row_tiles * 256;
    x.w0 = 0;
  }
  return x;
}

template <bool GROUPED>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_pair_rows_kernel(const __grid_constant__ CUtensorMap tmW,
                          const __grid_constant__ CUtensorMap tmA, const Args p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t full_bar[kStages], empty_bar[kStages], tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_slot, list[GROUPED ? kMaxList : 1];
  __shared__ int list_len;
  __shared__ volatile uint32_t abort_word, epi_abort;
  volatile uint32_t* abort_flag = &abort_word;

  grid_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();                  // 0 = leader
  const int pair_id = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 2);                           // one producer per CTA
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], 16);                        // eight epilogue warps of each CTA
    }
    abort_word = 0u;
    epi_abort = 0u;
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmA);
  }
  if (GROUPED && warp == 2) {
    // tiles of up to two neighbouring row tiles of an expert, (first tile << 16) + rows in use
    const int n = *p.num_rows / 128;
    int len = 0, odd = 0;                // odd: tiles of lane 0's expert in front of it, modulo 2
    for (int base = 0; base < n; base += 32) {
      const int t = base + lane;
      int e = -1, used = 0;
      bool start = false;
      if (t < n) {
        e = p.expert_ids[t];
        start = t == 0 || p.expert_ids[t - 1] != e;
        used = p.tile_rows[t];
        if (t + 1 < n && p.expert_ids[t + 1] == e) used += p.tile_rows[t + 1];
      }
      const unsigned int up_to = (2u << lane) - 1u;
      const unsigned int starts = __ballot_sync(0xffffffffu, start) & up_to;
      const int before = starts != 0u ? lane - (31 - __clz(starts)) : lane + odd;
      const bool keep = e >= 0 && (before & 1) == 0;
      const unsigned int vote = __ballot_sync(0xffffffffu, keep);
      const int at = len + __popc(vote & (up_to >> 1));
      if (keep && at < kMaxList) list[at] = (static_cast<uint32_t>(t) << 16) | static_cast<uint32_t>(used);
      len += __popc(vote);
      odd = (__shfl_sync(0xffffffffu, before, 31) + 1) & 1;
    }
    if (lane == 0) list_len = min(len, kMaxList);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // the other CTA's barriers exist before anything arrives there
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  grid_release();
  const int num_kb = (p.K + 63) / 64;
  const int units = (GROUPED ? list_len : p.row_tiles) * ((p.N + 255) / 256);

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = pair_id; ok && u < units; u += num_pairs) {
        const Unit x = unit_at<GROUPED>(p, list, u);
        const int half = x.rows / 2;
        const uint32_t bytes = kWBytes + half * 128;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, p.status, kKernelId, 0x100u + stage,
                         abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* sw = smem + stage * kStageBytes;
          const uint32_t full_leader = map_to_cta(&full_bar[stage], 0);
          mbar_expect_tx_remote(full_leader, bytes);
          tma_load_2d_pair(sw, &tmW, full_leader, kb * 64, x.w0 + x.n0 + static_cast<int>(rank) * kHalfW);
          const int m = x.m0 + static_cast<int>(rank) * half;
          if constexpr (GROUPED) {
            for (int r = 0; r < half; r += 16)
              tma_load_2d_pair(sw + kWBytes + r * 128, &tmA, full_leader, kb * 64, m + r);
          } else {
            tma_load_2d_pair(sw + kWBytes, &tmA, full_leader, kb * 64, m);
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      int stage = 0, it = 0;
      uint32_t phase = 0, tphase[2] = {0u, 0u};
      bool ok = true;
      for (int u = pair_id; ok && u < units; u += num_pairs, ++it) {
        const int b = it & 1;
        if (!mbar_wait(&tempty_bar[b], tphase[b] ^ 1u, p.status, kKernelId, 0x300u + b, abort_flag))
          break;
        tphase[b] ^= 1u;
        tc_fence_after();
        const uint32_t idesc = make_idesc(256, unit_at<GROUPED>(p, list, u).rows, 1, 1);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, p.status, kKernelId, 0x310u + stage, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sw = smem_u32(smem + stage * kStageBytes);
          const uint64_t wdesc = make_desc_k_sw128(sw), adesc = make_desc_k_sw128(sw + kWBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16_pair(tmem + static_cast<uint32_t>(b * kMaxRows),
                          wdesc + static_cast<uint64_t>(k * 2), adesc + static_cast<uint64_t>(k * 2),
                          idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit_pair(&empty_bar[stage]);              // frees the stage in both CTAs
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        umma_commit_pair(&tfull_bar[b]);                    // accumulators ready in both CTAs
      }
    }
  } else {
    // ---------------- epilogue: this CTA's 128 weight rows, 32 activation rows at a time ----------------
    // Two sets of four warps take the chunks of 32 rows in turn.  A lane holds 32 rows of one column: two
    // neighbours exchange one number for every two rows, and each stores two columns of one of them.
    const int q = warp & 3, set = (warp - 2) >> 2;
    uint32_t tphase[2] = {0u, 0u};
    const uint32_t tempty_leader[2] = {map_to_cta(&tempty_bar[0], 0), map_to_cta(&tempty_bar[1], 0)};
    const bool gated = p.epi == kSiluMul || p.epi == kGeluMul;
    const bool odd_lane = (lane & 1) != 0;
    // gate and up rows of the weights alternate in blocks of 32: of the lanes in quarters q and q ^ 1.  The
    // first takes the first 16 rows of a chunk, the second the others.
    const bool up = (q & 1) != 0;
    const int pair_bar = 2 + set * 2 + (q >> 1);
    float* xch = reinterpret_cast<float*>(smem + kOffOut) + (set * 2 + (q >> 1)) * 1024 + lane;
    int it = 0;
    for (int u = pair_id; u < units; u += num_pairs, ++it) {
      const int b = it & 1;
      const Unit x = unit_at<GROUPED>(p, list, u);
      const int n0 = x.n0 + static_cast<int>(rank) * kHalfW;
      if (!mbar_wait_warp(&tfull_bar[b], tphase[b], p.status, kKernelId, 0x400u + b, abort_flag))
        epi_abort = 1u;
      // (the warps meet at barriers below, so they leave together)
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (epi_abort != 0u) break;
      tphase[b] ^= 1u;
      tc_fence_after();
      // first of the lane's two columns
      const int col = (gated ? (n0 >> 1) + (q >> 1) * 32 : n0 + q * 32) + (lane & ~1);
      const bool inside = col < (gated ? p.N >> 1 : p.N);
      float bias0 = 0.0f, bias1 = 0.0f;
      if (p.epi == kBias && inside) {
        bias0 = __bfloat162float(p.bias[col]);
        bias1 = __bfloat162float(p.bias[col + 1]);
      }
      const uint32_t acc = tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(b * kMaxRows);
      bool released = false;
      for (int c = set * 32; c < x.used; c += 64) {
        uint32_t r[32];
        tmem_ld_32x32(acc + c, r);
        float scales = 1.0f;             // of row c + lane
        if (GROUPED && p.row_scale != nullptr && c + lane < x.used)
          scales = p.row_scale[x.m0 + c + lane];
        tmem_ld_wait();
        if (c + 64 >= x.used) {          // the set's last chunk is out of tensor memory
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(tempty_leader[b]);
          released = true;
        }
        if (gated) {
          pair_sync(pair_bar);       // the last chunk has been read
#pragma unroll
          for (int i = 0; i < 16; ++i) xch[(up ? 0 : 512) + i * 32] = __uint_as_float(up ? r[i] : r[16 + i]);
          pair_sync(pair_bar);
          float f[16], g[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float own = __uint_as_float(up ? r[16 + i] : r[i]), other = xch[(up ? 512 : 0) + i * 32];
            g[i] = up ? other : own;
            f[i] = up ? own : other;
          }
          if (p.epi == kSiluMul) {
#pragma unroll
            for (int i = 0; i < 16; ++i) f[i] = gated_f<false>(g[i], f[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) f[i] = gated_f<true>(g[i], f[i]);
          }
          const int row = c + (up ? 16 : 0) + (odd_lane ? 1 : 0);
          __nv_bfloat16* dst = p.C + static_cast<long long>(x.m0 + row) * p.ldc + col;
#pragma unroll
          for (int i = 0; i < 16; i += 2, dst += 2 * p.ldc) {
            const float in = __shfl_xor_sync(0xffffffffu, odd_lane ? f[i] : f[i + 1], 1);
            if (inside && row + i < x.used)
              *reinterpret_cast<uint32_t*>(dst) =
                  odd_lane ? pack_bf16x2(in, f[i + 1]) : pack_bf16x2(f[i], in);
          }
          continue;
        }
        const int row = c + (odd_lane ? 1 : 0);
        __nv_bfloat16* dst = p.C + static_cast<long long>(x.m0 + row) * p.ldc + col;
        // (a loop for each activation: one with the choice inside takes 170 cycles a turn)
        auto out = [&](auto act) {
          float lo[16], hi[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a0 = __uint_as_float(r[2 * i]), a1 = __uint_as_float(r[2 * i + 1]);
            const float in = __shfl_xor_sync(0xffffffffu, odd_lane ? a0 : a1, 1);
            lo[i] = odd_lane ? in : a0;
            hi[i] = odd_lane ? a1 : in;
            if (GROUPED) {
              const float s = __shfl_sync(0xffffffffu, scales, 2 * i + (odd_lane ? 1 : 0));
              lo[i] *= s;
              hi[i] *= s;
            }
          }
#pragma unroll
          for (int i = 0; i < 16; ++i, dst += 2 * p.ldc)
            if (inside && row + 2 * i < x.used)
              *reinterpret_cast<uint32_t*>(dst) = pack_bf16x2(act(lo[i]) + bias0, act(hi[i]) + bias1);
        };
        if (p.epi == kRelu2) out([](float v) { return relu2_f(v); });
        else if (p.epi == kGelu) out([](float v) { return gelu_f(v); });
        else out([](float v) { return v; });
      }
      if (!released) {                   // a tile of up to 32 rows: nothing for the second set
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(tempty_leader[b]);
      }
    }
  }
  // Nobody leaves before both CTAs are past their last MMA, commit and remote arrive.
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <bool GROUPED>
static int launch(const CUtensorMap& tmW, const CUtensorMap& tmA, Args a, int units,
                  cudaStream_t stream) {
  auto kernel = gemm_pair_rows_kernel<GROUPED>;
  static int at_once[64] = {0};            // pairs of SMs, per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -20;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * 74);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (at_once[dev] == 0) {
    cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    int n = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    at_once[dev] = e == cudaSuccess && n > 0 ? n : -1;
  }
  if (at_once[dev] < 0) return -20;
  a.status = status_ptr();
  cfg.gridDim = dim3(2 * (units < at_once[dev] ? units : at_once[dev]));
  cfg.stream = stream;
  cfg.numAttrs = 2;
  return launch_code(cudaLaunchKernelEx(&cfg, kernel, tmW, tmA, a));
}

static int make_maps(const void* W, uint64_t w_rows, long long ldw, const void* A, uint64_t a_rows,
                     long long lda, int K, int a_box, CUtensorMap* tmW, CUtensorMap* tmA) {
  int r = encode_tmap_2d(tmW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, W, w_rows, static_cast<uint64_t>(K),
                         static_cast<uint64_t>(ldw) * 2, kHalfW, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r == 0)
    r = encode_tmap_2d(tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, a_rows, static_cast<uint64_t>(K),
                       static_cast<uint64_t>(lda) * 2, a_box, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  return r < 0 ? -6 : r;
}

}  // namespace pair_rows
}  // namespace b200

// C[M, N] = A[M, K] * W[N, K]^T in as few tiles of at most `rows` activation rows as there can
// be, of one size (a multiple of 32, at most 256; 0: 256).  Constraints and epilogues as b200_gemm_stream,
// without fp32 results.  -20: not covered.
B200_API int b200_gemm_pair_rows(const void* A, long long lda, const void* W, long long ldw, void* C,
                                 long long ldc, int M, int N, int K, const void* bias, int epi, int rows,
                                 void* stream) {
  using namespace b200;
  using namespace b200::pair_rows;
  if (M <= 0 || N <= 0) return 0;
  const bool gated = epi == kSiluMul || epi == kGeluMul;
  if (!(gated || epi == kNone || epi == kBias || epi == kRelu2 || epi == kGelu) ||
      (gated && (N % 64) != 0) || rows < 0 || rows > kMaxRows || (rows % 32) != 0)
    return -20;
  if (K <= 0 || (K % 8) != 0 || (N % 8) != 0 || (lda % 8) != 0 || (ldw % 8) != 0 || (ldc % 8) != 0)
    return -2;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) |
       reinterpret_cast<uintptr_t>(C)) & 15)
    return -3;
  if (epi == kBias && bias == nullptr) return -5;
  Args a = {};
  if (rows == 0) rows = kMaxRows;
  a.row_tiles = (M + rows - 1) / rows;
  a.rows = ((M + a.row_tiles - 1) / a.row_tiles + 31) / 32 * 32;
  a.row_tiles = (M + a.rows - 1) / a.rows;
  CUtensorMap tmW, tmA;
  const int r = make_maps(W, N, ldw, A, M, lda, K, a.rows / 2, &tmW, &tmA);
  if (r != 0) return r;
  a.C = static_cast<__nv_bfloat16*>(C);
  a.ldc = ldc;
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.M = M; a.N = N; a.K = K;
  a.epi = epi;
  return launch<false>(tmW, tmA, a, (N + 255) / 256 * a.row_tiles, static_cast<cudaStream_t>(stream));
}

// Experts: as b200_gemm_stream_grouped, with the rows in use of every row tile (tile_rows [M_cap / 128])
// in place of the sorted ids.  -20: not covered.
B200_API int b200_gemm_pair_rows_grouped(const void* A, long long lda, const void* W, long long ldw,
                                         void* C, long long ldc, int M_cap, int N, int K, int E,
                                         const int* expert_ids, const int* num_rows,
                                         const int* tile_rows, const float* row_scale, int epi,
                                         void* stream) {
  using namespace b200;
  using namespace b200::pair_rows;
  if (M_cap <= 0 || N <= 0 || E <= 0) return 0;
  if ((M_cap % 128) != 0 || K <= 0 || (K % 8) != 0 || (lda % 8) != 0 || (ldw % 8) != 0 ||
      (ldc % 8) != 0 || expert_ids == nullptr || num_rows == nullptr || tile_rows == nullptr)
    return -2;
  // (every expert has at most one tile that is not paired)
  if ((N % 64) != 0 || (epi != kNone && epi != kSiluMul && epi != kRelu2 && epi != kGelu) ||
      (M_cap / 128 + E + 1) / 2 > kMaxList)
    return -20;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) |
       reinterpret_cast<uintptr_t>(C)) & 15)
    return -20;
  CUtensorMap tmW, tmA;
  const int r = make_maps(W, static_cast<uint64_t>(E) * N, ldw, A, M_cap, lda, K, 16, &tmW, &tmA);
  if (r != 0) return r;
  Args a = {};
  a.C = static_cast<__nv_bfloat16*>(C);
  a.ldc = ldc;
  a.M = M_cap; a.N = N; a.K = K;
  a.epi = epi;
  a.expert_ids = expert_ids; a.num_rows = num_rows; a.tile_rows = tile_rows; a.row_scale = row_scale;
  return launch<true>(tmW, tmA, a, M_cap / 128 * ((N + 255) / 256), static_cast<cudaStream_t>(stream));
}
