// Weight-only quantised GEMM for decode-sized activations:
//   C[M, N] = A[M, K] * dequant(W)[N, K]^T,  M <= 256, W stored as 4-bit or 8-bit integers with
// per-group scales: w = q * scale - zs (zs = zero point * scale), groups of g along K.
//
// Replaces the reference's `gptq_gemm` / `awq_gemm` ops on the decode path
// (vllm_gcu/kernels/quantization/awq.py:70-118, gptq.py:95-164).  The layer is bound by its packed
// bytes (4 bit: 0.53 bytes a weight) and, close behind, by the instructions that de-quantise them:
// 4.75 per pair of weights, 14 us for the 218 M weights of a Llama-3-8B layer on 148 SMs, 17 us for
// their bytes at copy bandwidth.
//
// The operands are swapped, as in gemm_stream.cu: 128 weight rows are the M side of tcgen05.mma and the
// activation rows its N side.  TMA brings packed tiles of 128 rows x 128 bytes into a ring; a thread
// owns one weight row, de-quantises 64 of its weights in registers (4 bit: bf16 pair arithmetic with a
// single rounding) and stores them into tensor memory, from where tcgen05.mma takes its A operand: no
// shared-memory stores and no proxy fence per tile, which held the former kernel (bf16 tiles of 64 x 64
// built in shared memory) at 0.3 us a tile.  Activations come by TMA into a ring of their own.  K is
// split over a cluster of CTAs that add their partial sums through shared memory (stream.cuh).
//
// Roles (384 threads): warp 0 TMA of packed weights, warp 1 tcgen05.mma, warp 2 TMA of activations,
// warp 3 owner of tensor memory, warps 4..7 and 8..11 de-quantise the first and second half of a packed tile
// (warp w can reach the lanes 32 (w mod 4) .. + 31); warps 4..7 move the accumulators out.  A buffer of
// de-quantised weights belongs to one group of warps: with a third group that shared them a warp could be two
// uses ahead of a barrier's parity.  Every wait is bounded.
#include "stream.cuh"

namespace b200 {
namespace wna16s {

using namespace b200::stream;

constexpr unsigned int kKernelId = 71;
constexpr int kThreads = 384;
constexpr int kPackedBytes = BW * 128;   // a packed tile
constexpr int kMaxPacked = 8, kMaxX = 16;
constexpr int kEarlyRows = 64;           // see the kernel
constexpr int kACols = 128;              // columns of de-quantised weights in tensor memory

struct Args {
  const __nv_bfloat16* scales;    // [N, K / g]
  const __nv_bfloat16* zs;        // [N, K / g]
  const __nv_bfloat16* bias;      // optional [N]
  __nv_bfloat16* C;
  long long ldc;
  int M, N, K, g_shift;
  int rows;                       // activation rows of a tile, a multiple of 16
  int row_tiles;
  int splits, packed_stages, x_stages;
  unsigned int* status;
};

// 8 nibbles, low one first -> 4 bf16 pairs q * s - z.  A byte permute brings a byte's two nibbles to
// the low ends of two halves; 0x4300 | q is the bf16 number 128 + q, the subtraction of 128 is exact and
// the fused multiply-add rounds once.  (The integer pipe, half as wide as the others, is what bounds the
// kernel: nine of these instructions a word here, eleven when four shifts and masks give the pairs
// (0, 4), (1, 5), (2, 6), (3, 7) and four permutes restore the order.)
__device__ __forceinline__ void dequant8(uint32_t q, __nv_bfloat162 s2, __nv_bfloat162 nz2,
                                         uint32_t* w) {
  const __nv_bfloat162 k128 = __float2bfloat162_rn(128.0f);
  const uint32_t high = q >> 4;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t bits =
        (__byte_perm(q, high, 0x4400u + 0x1111u * j) & 0x000F000Fu) | 0x43004300u;
    const __nv_bfloat162 v =
        __hfma2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&bits), k128), s2, nz2);
    w[j] = *reinterpret_cast<const uint32_t*>(&v);
  }
}

// SMALL: layers of few packed tiles, whose rows may be dealt out over blockIdx.z.  They, and tiles of up to
// kEarlyRows rows, set up and bring their first packed tiles into L2 before they wait for the kernel in
// front (12 rows, the four products of a layer 76.8 -> 73.4 us); with 128 rows a kernel that already holds its place takes issue
// slots from the de-quantising warps of the one in front (93.1 : 95.1).
// VEC: the scales of eight groups of 128 come in one 16-byte load, a row a lane.  One by one, a row's
// scales lie in lines that do not stay in what the ring leaves of the cache, and as many bytes of them as
// of weights came from L2 (96 rows, the four products of a layer 96.2 -> 88.3 us, 12 rows 82.8 -> 76.8).
template <int BITS, bool SMALL, bool VEC>
__global__ void __launch_bounds__(kThreads, 2)
    gemm_wna16_stream_kernel(const __grid_constant__ CUtensorMap tmW,
                             const __grid_constant__ CUtensorMap tmA, const Args p) {
  // A step is half a packed tile, 64 bytes of every row: one or two blocks of 64 weights.  The two groups
  // of de-quantising warps take the steps in turn, each with buffers of its own.
  constexpr int kBlocks = BITS == 4 ? 2 : 1;          // blocks of a step
  constexpr int kVec = BITS == 4 ? 2 : 4;             // 16-byte words of a row in a block
  constexpr int kBufs = kACols / (32 * kBlocks);      // steps in tensor memory
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* smem_x = smem + p.packed_stages * kPackedBytes;
  const int x_block = p.rows * 128, x_bytes = kBlocks * x_block;
  __shared__ uint64_t pfull[kMaxPacked], pempty[kMaxPacked], xfull[kMaxX], xempty[kMaxX];
  __shared__ uint64_t afull[kBufs], aempty[kBufs], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile uint32_t abort_word;
  volatile uint32_t* abort_flag = &abort_word;

  const bool early = SMALL || p.rows <= kEarlyRows;
  if (!early) grid_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = static_cast<int>(blockIdx.x);
  const int n0 = static_cast<int>(blockIdx.y) * BW;
  const int m0 = SMALL ? static_cast<int>(blockIdx.z) * p.rows : 0;
  const int used = SMALL ? min(p.M - m0, p.rows) : p.M;
  uint32_t acc_cols = 32;
  while (acc_cols < static_cast<uint32_t>(p.rows)) acc_cols <<= 1;
  const uint32_t cols = acc_cols <= 128 ? 256 : 512;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.packed_stages; ++s) {
      mbar_init(&pfull[s], 1);
      mbar_init(&pempty[s], 8);           // one arrival of every de-quantising warp
    }
    for (int s = 0; s < p.x_stages; ++s) {
      mbar_init(&xfull[s], 1);
      mbar_init(&xempty[s], 1);
    }
    for (int s = 0; s < kBufs; ++s) {
      mbar_init(&afull[s], 4);
      mbar_init(&aempty[s], 1);
    }
    mbar_init(&done_bar, 1);
    abort_word = 0u;
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmA);
  }
  if (warp == 3) {
    tmem_alloc(&tmem_slot, cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot, tmem_a = tmem + acc_cols;

  // this CTA's packed tiles, and its blocks of 64 (the last tile of a row may hold fewer)
  const int total_blocks = p.K / 64;
  const int total_tiles = (total_blocks + 2 * kBlocks - 1) / (2 * kBlocks);
  const int t_lo = static_cast<int>(static_cast<long long>(split) * total_tiles / p.splits);
  const int t_hi = static_cast<int>(static_cast<long long>(split + 1) * total_tiles / p.splits);
  const int b_lo = t_lo * 2 * kBlocks;
  const int blocks = min(t_hi * 2 * kBlocks, total_blocks) - b_lo;
  const int steps = (blocks + kBlocks - 1) / kBlocks;
  if (early) {
    // the first packed tiles come into L2 while the kernels in front still run
    if (threadIdx.x == 0)
      for (int t = t_lo; t < t_hi && t < t_lo + p.packed_stages; ++t) tma_prefetch_2d(&tmW, t * 128, n0);
    __syncwarp();
    grid_wait();
  }

  if (warp == 0) {
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 0;
      for (int t = t_lo; t < t_hi; ++t) {
        if (!mbar_wait(&pempty[s], phase ^ 1u, p.status, kKernelId, 0x100u + s, abort_flag)) break;
        mbar_expect_tx(&pfull[s], kPackedBytes);
        tma_load_2d(smem + s * kPackedBytes, &tmW, &pfull[s], t * 128, n0);
        if (++s == p.packed_stages) {
          s = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 2) {
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 0;
      for (int b = 0; b < blocks; b += kBlocks) {
        if (!mbar_wait(&xempty[s], phase ^ 1u, p.status, kKernelId, 0x200u + s, abort_flag)) break;
        const int n = min(kBlocks, blocks - b);
        mbar_expect_tx(&xfull[s], n * x_block);
        for (int i = 0; i < n; ++i)
          tma_load_2d(smem_x + s * x_bytes + i * x_block, &tmA, &xfull[s], (b_lo + b + i) * 64, m0);
        if (++s == p.x_stages) {
          s = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc(BW, p.rows, 1, 1);
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int st = 0; st < steps; ++st) {
        const int buf = st % kBufs;
        if (!mbar_wait(&xfull[s], phase, p.status, kKernelId, 0x300u + s, abort_flag) ||
            !mbar_wait(&afull[buf], static_cast<uint32_t>(st / kBufs) & 1u, p.status, kKernelId,
                       0x320u + buf, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t xdesc = make_desc_k_sw128(smem_u32(smem_x + s * x_bytes));
        const uint32_t ta = tmem_a + buf * (32 * kBlocks);
#pragma unroll
        for (int i = 0; i < kBlocks; ++i) {
          if (i > 0 && st * kBlocks + i >= blocks) break;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16_ts(tmem, ta + i * 32 + k * 8,
                        xdesc + static_cast<uint32_t>(i * (x_block >> 4) + k * 2), idesc,
                        (st > 0 || i > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&xempty[s]);
        umma_commit(&aempty[buf]);
        if (++s == p.x_stages) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (ok) umma_commit(&done_bar);
    }
  } else if (warp >= 4) {
    const int q = warp & 3, group = (warp - 4) >> 2;
    const int row = q * 32 + lane, n = n0 + row;
    const uint32_t lane_addr = tmem_a + (static_cast<uint32_t>(q * 32) << 16);
    const long long groups = p.K >> p.g_shift;
    // rows past N hold zeros and are never stored: any scale will do
    const __nv_bfloat16* srow = p.scales + (n < p.N ? n : 0) * groups;
    const __nv_bfloat16* zrow = p.zs + (n < p.N ? n : 0) * groups;
    const bool halves = !VEC && p.g_shift < 6;        // groups of 32: two per block
    // Scales of the next step.  VEC: groups of 128, one per step, so that the two groups of warps take the two
    // halves of each 32-bit word of a row's scales: eight groups in one 16-byte load, a word a step.
    __nv_bfloat16 sc[VEC ? 1 : 2 * kBlocks], zz[VEC ? 1 : 2 * kBlocks];
    uint4 s8, z8;
    int word = 0;
    auto fetch = [&](int st) {
      if constexpr (VEC) {
        const int g8 = (t_lo + (st >> 1)) >> 2;          // (a packed tile is two groups)
        s8 = reinterpret_cast<const uint4*>(srow)[g8];
        z8 = reinterpret_cast<const uint4*>(zrow)[g8];
      } else {
#pragma unroll
        for (int i = 0; i < kBlocks; ++i) {
          const int b = min(st * kBlocks + i, blocks - 1);
          const int g0 = ((b_lo + b) * 64) >> p.g_shift;
          sc[2 * i] = srow[g0];
          zz[2 * i] = zrow[g0];
          if (halves) {
            sc[2 * i + 1] = srow[g0 + 1];
            zz[2 * i + 1] = zrow[g0 + 1];
          }
        }
      }
    };
    if (group < steps) fetch(group);
    if constexpr (VEC) word = t_lo & 3;
    int s = 0;
    uint32_t phase = 0;
    for (int st = group; st < steps; st += 2) {
      mbar_pass_warp(&pfull[s], phase, p.status, kKernelId, 0x400u + s, abort_flag);
      const uint8_t* tile = smem + s * kPackedBytes + row * 128;
      const int buf = st % kBufs;
      __nv_bfloat162 s2[2 * kBlocks], nz2[2 * kBlocks];
      if constexpr (VEC) {
        const uint32_t sw = word < 2 ? (word == 0 ? s8.x : s8.y) : (word == 2 ? s8.z : s8.w);
        const uint32_t zw = word < 2 ? (word == 0 ? z8.x : z8.y) : (word == 2 ? z8.z : z8.w);
        const uint32_t pick = group == 0 ? 0x1010u : 0x3232u;
        const uint32_t sb = __byte_perm(sw, 0u, pick), zb = __byte_perm(zw, 0u, pick) ^ 0x80008000u;
#pragma unroll
        for (int h = 0; h < 2 * kBlocks; ++h) {
          s2[h] = *reinterpret_cast<const __nv_bfloat162*>(&sb);
          nz2[h] = *reinterpret_cast<const __nv_bfloat162*>(&zb);
        }
      } else {
#pragma unroll
        for (int h = 0; h < 2 * kBlocks; ++h) {
          s2[h] = __bfloat162bfloat162((h & 1) == 1 && halves ? sc[h] : sc[h & ~1]);
          nz2[h] = __hneg2(__bfloat162bfloat162((h & 1) == 1 && halves ? zz[h] : zz[h & ~1]));
        }
      }
      uint4 u[4];
#pragma unroll
      for (int v = 0; v < 4; ++v)
        u[v] = *reinterpret_cast<const uint4*>(tile + (((group * 4 + v) ^ (row & 7)) << 4));
      if constexpr (VEC) {
        if (++word == 4) {
          word = 0;
          if (st + 2 < steps) fetch(st + 2);
        }
      } else if (st + 2 < steps) {
        fetch(st + 2);
      }
#pragma unroll
      for (int i = 0; i < kBlocks; ++i) {
        uint32_t w[32];
#pragma unroll
        for (int v = 0; v < kVec; ++v) {
          const uint4 x4 = u[i * kVec + v];
          const uint32_t words[4] = {x4.x, x4.y, x4.z, x4.w};
          if constexpr (BITS == 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) dequant8(words[j], s2[i * 2 + v], nz2[i * 2 + v], w + v * 16 + j * 4);
          } else {
            const float fs = __bfloat162float(s2[v >> 1].x), fz = __bfloat162float(nz2[v >> 1].x);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t x = words[j];
              w[v * 8 + j * 2] = pack_bf16x2(fmaf(static_cast<float>(x & 0xFFu), fs, fz),
                                             fmaf(static_cast<float>((x >> 8) & 0xFFu), fs, fz));
              w[v * 8 + j * 2 + 1] = pack_bf16x2(fmaf(static_cast<float>((x >> 16) & 0xFFu), fs, fz),
                                                 fmaf(static_cast<float>(x >> 24), fs, fz));
            }
          }
        }
        if (i == 0) {
          mbar_pass_warp(&aempty[buf], (static_cast<uint32_t>(st / kBufs) & 1u) ^ 1u, p.status, kKernelId,
                         0x420u + buf, abort_flag);
          tc_fence_after();
        }
        tmem_st_32x32(lane_addr + buf * (32 * kBlocks) + i * 32, w);
      }
      // the packed words are in registers: both barriers of the step at once
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&afull[buf]);
        mbar_arrive(&pempty[s]);
      }
      if (++s == p.packed_stages) {
        s = 0;
        phase ^= 1u;
      }
    }
    // (a last packed tile of one step: the other group has nothing to wait for)
    __syncwarp();
    // every ring slot has been consumed when done_bar completes, so the partial sums take their place
    // (the other de-quantising group has read its last packed tile before its last block was multiplied)
    if (group == 0) {
      const bool ok = mbar_wait_warp(&done_bar, 0u, p.status, kKernelId, 0x500u, abort_flag);
      // Not earlier: a next kernel that already holds its place takes issue slots from the de-quantising
      // warps (96 requests over eight layers 1642 us with the release in front, 1553 here, 1567 without).
      grid_release();
      __syncwarp();
      tc_fence_after();
      if (ok) park_sums(tmem, reinterpret_cast<float*>(smem), q, lane, used);
    }
  }
  tc_fence_before();
  if (p.splits > 1) cluster_arrive_wait();
  else __syncthreads();
  if (abort_word == 0u)
    sum_rows<false, false>(smem, split, p.splits, warp, kThreads / 32, lane, used, [&](int r, float4 v) {
      const int col = n0 + 4 * lane;
      __nv_bfloat16* out = p.C + static_cast<long long>(m0 + r) * p.ldc + col;
      float f[4] = {v.x, v.y, v.z, v.w};
      if (col + 4 <= p.N && (p.ldc & 3) == 0) {
        if (p.bias != nullptr)
#pragma unroll
          for (int i = 0; i < 4; ++i) f[i] += __bfloat162float(p.bias[col + i]);
        *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
        return;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (col + i < p.N)
          out[i] = __float2bfloat16(
              f[i] + (p.bias != nullptr ? __bfloat162float(p.bias[col + i]) : 0.0f));
    });
  // nobody leaves while another CTA may still read its partial sums
  if (p.splits > 1) cluster_arrive_wait();
  else __syncthreads();
  if (warp == 3) tmem_dealloc(tmem, cols);
}

template <int BITS>
static int launch(const void* A, long long lda, const void* qw, Args a, cudaStream_t stream) {
  const int tiles = (a.N + BW - 1) / BW;
  const int packed = (a.K / 64 + (BITS == 4 ? 3 : 1)) / (BITS == 4 ? 4 : 2);
  const bool small = packed <= 8;
  // scales of eight groups of 128 in 16 bytes, every row from a boundary
  const bool vec = BITS == 4 && a.g_shift == 7 && (a.K & 1023) == 0 &&
                   ((reinterpret_cast<uintptr_t>(a.scales) | reinterpret_cast<uintptr_t>(a.zs)) & 15) == 0;
  static AtOnce table[4] = {};
  constexpr bool kVec = BITS == 4;
  auto kernel = small ? (vec ? gemm_wna16_stream_kernel<BITS, true, kVec> : gemm_wna16_stream_kernel<BITS, true, false>)
                : vec ? gemm_wna16_stream_kernel<BITS, false, kVec>
                      : gemm_wna16_stream_kernel<BITS, false, false>;
  const int* at_once = clusters_at_once(table[small + 2 * vec], kernel, kThreads);
  if (at_once == nullptr) return -20;
  // Bound by the de-quantising warps, so what counts is that every SM has the same share: two CTAs per
  // SM and the largest split that one wave takes, down to two packed tiles a slice (four above 32 rows,
  // where the sums of a slice cost more).  4096 x 14336 at 16 rows: eight slices 22.7 us, four 25.2; at
  // 128 rows 29.2 and 29.5; 4096 x 4096 at 128 rows: eight 16.6, four 14.4; 6144 x 4096 at 16 rows in
  // one wave (five) 15.0, in two (six) 19.5.  Above 128 rows accumulators and de-quantised blocks fill
  // the tensor memory of an SM: one CTA.
  a.row_tiles = 1;
  a.rows = (a.M + 15) / 16 * 16;
  a.splits = 1;
  for (int s = 2; s <= kMaxSplits; ++s)
    if (packed >= s * (a.rows > 32 ? 4 : 2) && tiles <= at_once_for(at_once, s, a.rows > 128 ? 1 : 2))
      a.splits = s;
  // Layers of few packed tiles leave most SMs idle that way.  With one CTA per SM a slice may have as
  // little as one packed tile, and the rows may be dealt out as well (every tile de-quantises for itself):
  // a CTA takes about as long for a packed tile, 1 us, as for moving out the sums of 50 rows, and two on an SM
  // 1.7 times as long as one.  4 bits, one tile of rows and slices as above : as here (tiles of 64 x 64 built in
  // shared memory), us: 64 x 512 x 512 7.7 : 4.9 (6.4), 256 x 512 x 512 12.6 : 5.0 (8.1), 256 x 1024 x
  // 1024 15.5 : 6.4 (11.0), 128 x 4096 x 1024 12.0 : 7.7 (9.2), 256 x 2048 x 2048 15.0 : 9.2 (23).
  if (small) {
    auto cost = [&](int row_tiles, int rows, int splits) {
      const int load = (tiles * row_tiles * splits + at_once[1] - 1) / at_once[1];
      return ((packed + splits - 1) / splits + rows * 0.02) * (load > 1 ? 0.85 * load : 1.0);
    };
    double best = cost(1, a.rows, a.splits);
    for (int t = 1; t <= 16; t *= 2) {
      const int rows = ((a.M + t - 1) / t + 15) / 16 * 16;
      for (int s = 1; s <= kMaxSplits && s <= packed; ++s)
        if (tiles * t <= at_once[s] && cost(t, rows, s) < best) {
          best = cost(t, rows, s);
          a.rows = rows;
          a.splits = s;
        }
    }
    a.row_tiles = (a.M + a.rows - 1) / a.rows;
  }
  const int per_sm = a.rows > 128 ? 1 : 2;
  a.packed_stages = per_sm == 2 ? 2 : 6;
  const int room = (per_sm == 2 ? kSmemLimit / 2 - 1024 : kSmemLimit) - 1024;
  const int step = BITS == 4 ? 2 : 1;           // blocks of activations in a stage
  a.x_stages = (room - a.packed_stages * kPackedBytes) / (a.rows * 128 * step);
  if (a.x_stages > kMaxX) a.x_stages = kMaxX;
  const int ring = a.packed_stages * kPackedBytes + a.x_stages * a.rows * 128 * step;
  const int sums = a.rows * BW * 4;
  const int bytes = (ring > sums ? ring : sums) + 1024;
  if (a.x_stages < 2 || bytes > kSmemLimit) return -20;
  const uint64_t kbytes = static_cast<uint64_t>(BITS == 4 ? a.K / 2 : a.K);
  CUtensorMap tmW, tmA;
  int r = encode_tmap_2d(&tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, qw, static_cast<uint64_t>(a.N), kbytes,
                         kbytes, BW, 128, CU_TENSOR_MAP_SWIZZLE_128B);
  if (r == 0)
    r = encode_tmap_2d(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, static_cast<uint64_t>(a.M),
                       static_cast<uint64_t>(a.K), static_cast<uint64_t>(lda) * 2, a.rows, 64,
                       CU_TENSOR_MAP_SWIZZLE_128B);
  if (r != 0) return r < 0 ? -6 : r;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = launch_config(a.splits, tiles, kThreads, bytes, attr, stream);
  cfg.gridDim.z = a.row_tiles;
  return launch_code(cudaLaunchKernelEx(&cfg, kernel, tmW, tmA, a));
}

}  // namespace wna16s
}  // namespace b200

// A [M, K] bf16 (row pitch lda), qw [N, K / 2] (low nibble = even k) or [N, K] for 8 bit, scales / zs
// [N, K / g], C [M, N] bf16.  Returns -20 when the shape is outside what the kernel covers (M > 256,
// K % 64, group size not a power of two >= 32, misaligned pointers): callers de-quantise and use the
// bf16 GEMM.
B200_API int b200_gemm_wna16(const void* A, long long lda, const void* qw, const void* scales,
                             const void* zs, const void* bias, void* C, long long ldc, int M,
                             int N, int K, int g, int bits, void* stream) {
  using namespace b200;
  using namespace b200::wna16s;
  if (M <= 0 || N <= 0) return 0;
  if (M > 256 || K <= 0 || (K % 64) != 0 || g < 32 || (g & (g - 1)) != 0 || (K % g) != 0 ||
      (bits != 4 && bits != 8) || (lda % 8) != 0 ||
      ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(qw)) & 15))
    return -20;
  Args a;
  a.scales = static_cast<const __nv_bfloat16*>(scales);
  a.zs = static_cast<const __nv_bfloat16*>(zs);
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.C = static_cast<__nv_bfloat16*>(C);
  a.ldc = ldc;
  a.M = M; a.N = N; a.K = K;
  a.g_shift = 31 - __builtin_clz(static_cast<unsigned>(g));
  a.status = status_ptr();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return bits == 4 ? launch<4>(A, lda, qw, a, s) : launch<8>(A, lda, qw, a, s);
}
