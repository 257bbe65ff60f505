// Prefill attention of two query heads at once (included by attention_fmha.cu, whose Args and constants
// it uses): head dimension 128, heads in pairs over one key head, no soft cap, chunk or bias.
//
// What bounds it: per 128 x 128 scores the tensor cores need 1024 cycles (Q K^T and P V) and the
// exponentials 1024 cycles of the special-function pipe, so neither may wait for the other.  With one
// query tile a CTA runs scores -> softmax -> P V back to back (about 6000 cycles a tile).  Here a CTA
// holds the query tiles of two heads that read the same keys: while the softmax warps of one work, the
// tensor cores multiply for the other, and every key tile is loaded once for both.  Probabilities go
// back into the tensor memory that held the scores, from where P V takes them as its A operand: no
// shared-memory stores and no proxy fence in the chain.  One thread owns a row of 128 scores, read once
// into registers: no exchange of maxima.
//
// Order of the tensor-core work: S_a(0) S_b(0), then for every key tile j: P_a V(j), S_a(j + 1), P_b
// V(j), S_b(j + 1).  It executes in the order of issue, so the barrier that announces S(j) also says
// that P V(j - 1) has read its probabilities and finished its sums: the softmax warps may rescale the
// output in place without another wait.  The running maximum is raised only when it is exceeded by 8 in
// the log2 domain, as in the kernel for one head.
//
// Warps: 0 TMA (lane = page and half of a key tile), 1 tcgen05.mma and owner of tensor memory, 2..5
// softmax and epilogue of the first head, 6..9 of the second.  The longest query tiles start first.
#pragma once

namespace b200 {
namespace fmha {

constexpr int kPairSlots = 5;                     // key and value tiles in flight
constexpr int kPairOffRing = 2 * kTile;           // behind the two query tiles
constexpr int kPairOffBar = kPairOffRing + kPairSlots * kTile;
constexpr int kPairSmemBytes = kPairOffBar + 256 + 1024;
constexpr uint32_t kPairColO = 256;               // scores of head h: 128 h, outputs 256 + 128 h
static_assert(kPairSmemBytes <= 232448, "exceeds the shared memory of one CTA");

__global__ void __launch_bounds__(kThreads, 1)
    fmha_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const Args a) {
  constexpr int HD = 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kPairOffBar);
  uint64_t* q_full = bars;                  // 1
  uint64_t* full = bars + 1;                // ring of K(0) V(0) K(1) V(1) ...
  uint64_t* empty = full + kPairSlots;
  uint64_t* s_full = empty + kPairSlots;    // per head: scores are there
  uint64_t* p_full = s_full + 2;            // per head: probabilities are there, output rescaled
  uint64_t* o_done = p_full + 2;            // per head: the last product has finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  int* s_info = reinterpret_cast<int*>(tmem_slot + 2);   // [0] sequence, [1] q tile in sequence

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head0 = 2 * blockIdx.y;
  const int tile_x = static_cast<int>(gridDim.x - 1 - blockIdx.x);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < kPairSlots; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1);
    }
    *abort_flag = 0u;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 2) {
    int found, qt;
    find_tile(a, tile_x, lane, &found, &qt);
    if (lane == 0) {
      s_info[0] = found;
      s_info[1] = qt;
    }
  }
  __syncthreads();
  const int seq = s_info[0];
  if (seq < 0) return;                       // surplus CTA (grid is an upper bound)
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  const int q_start = a.cu_q[seq];
  const int q_len = a.cu_q[seq + 1] - q_start;
  const int seq_len = a.seq_lens[seq];
  const int q0 = s_info[1] * BQ;
  const int rows = min(BQ, q_len - q0);
  const int pos0 = seq_len - q_len + q0;                // absolute position of the tile's first row
  const int kv_hi = a.causal ? min(seq_len, pos0 + rows) : seq_len;
  const int kv_lo = a.window > 0 ? max(0, pos0 - a.window + 1) : 0;
  const int t0 = kv_lo / BKV;
  const int nt = (kv_hi + BKV - 1) / BKV - t0;          // >= 1
  const int kvh = head0 / (a.Hq / a.Hkv);

  if (warp == 0) {
    // ---------------- TMA: lane = (page of 16 keys, half of the head dimension) ----------------
    if (lane == 0) {
      mbar_expect_tx(q_full, 2 * kTile);
      for (int h = 0; h < 2; ++h)
        for (int c = 0; c < 2; ++c)
          tma_load_2d(smem + h * kTile + c * kSub, &tmQ, q_full, (head0 + h) * HD + c * 64,
                      q_start + q0);
    }
    const int* bt = a.block_tables + static_cast<long long>(seq) * a.max_blocks;
    const int last_tok = seq_len - 1;
    const int page = lane >> 1, half = lane & 1;
    int slot = 0;
    uint32_t phase = 0;
    for (int j = 0; j < nt; ++j) {
      const int key = (t0 + j) * BKV + page * kPage;
      int y = 0;
      if (lane < 2 * (BKV / kPage))          // pages past the end: any valid page
        y = bt[min(key, last_tok) / a.block_size] * a.block_size + key % a.block_size;
      bool ok = true;
      for (int kv = 0; kv < 2 && ok; ++kv) {
        ok = mbar_wait_warp(&empty[slot], phase ^ 1u, a.status, kKernelId, 0x600u + slot, abort_flag);
        if (ok) {
          if (lane == 0) mbar_expect_tx(&full[slot], kTile);
          __syncwarp();
          if (lane < 2 * (BKV / kPage))
            tma_load_2d(smem + kPairOffRing + slot * kTile + half * kSub + page * (kPage * 128),
                        kv == 0 ? &tmK : &tmV, &full[slot], kvh * HD + half * 64, y);
        }
        if (++slot == kPairSlots) {
          slot = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t kIdescS = make_idesc(BQ, BKV, 1, 1);
      constexpr uint32_t kIdescO = make_idesc(BQ, HD, 1, 1) | kIdescBMajorMN;
      const uint32_t q_addr = smem_u32(smem), ring = smem_u32(smem + kPairOffRing);
      // K(j) is entry 2 j of the ring, V(j) entry 2 j + 1
      auto wait_entry = [&](int e) {
        return mbar_wait(&full[e % kPairSlots], static_cast<uint32_t>(e / kPairSlots) & 1u, a.status,
                         kKernelId, 0x610u + e % kPairSlots, abort_flag);
      };
      auto issue_s = [&](int h, int j) {
        const uint32_t k_addr = ring + (2 * j) % kPairSlots * kTile;
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t sub = (ks >> 2) * kSub;
          umma_f16(tmem + h * BKV,
                   make_desc_k_sw128(q_addr + h * kTile + sub) + static_cast<uint64_t>((ks & 3) * 2),
                   make_desc_k_sw128(k_addr + sub) + static_cast<uint64_t>((ks & 3) * 2), kIdescS,
                   ks > 0 ? 1u : 0u);
        }
        umma_commit(&s_full[h]);
      };
      bool ok = mbar_wait(q_full, 0, a.status, kKernelId, 0x620u, abort_flag) && wait_entry(0);
      if (ok) {
        tc_fence_after();
        issue_s(0, 0);
        issue_s(1, 0);
        umma_commit(&empty[0]);
      }
      for (int j = 0; ok && j < nt; ++j) {
        ok = wait_entry(2 * j + 1);
        for (int h = 0; ok && h < 2; ++h) {
          ok = mbar_wait(&p_full[h], j & 1, a.status, kKernelId, 0x630u + h, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint64_t vdesc =
              make_desc_mn_sw128(ring + (2 * j + 1) % kPairSlots * kTile, kSub);
#pragma unroll
          for (int ks = 0; ks < BKV / 16; ++ks)
            umma_f16_ts(tmem + kPairColO + h * HD, tmem + h * BKV + ks * 8,
                        vdesc + static_cast<uint64_t>(ks) * (2048 >> 4), kIdescO,
                        (j > 0 || ks > 0) ? 1u : 0u);
          if (h == 1) umma_commit(&empty[(2 * j + 1) % kPairSlots]);
          if (j + 1 == nt) {
            umma_commit(&o_done[h]);
            continue;
          }
          if (h == 0) {
            ok = wait_entry(2 * j + 2);
            if (!ok) break;
            tc_fence_after();
          }
          issue_s(h, j + 1);
          if (h == 1) umma_commit(&empty[(2 * j + 2) % kPairSlots]);
        }
      }
    }
  } else {
    // ---------------- softmax + epilogue: one thread per query row ----------------
    const int h = (warp - 2) >> 2;
    const int qd = warp & 3;                    // TMEM lane quarter
    const int r = qd * 32 + lane;               // query row in the tile
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(qd * 32) << 16);
    const uint32_t s_addr = lane_addr + h * BKV, o_addr = lane_addr + kPairColO + h * HD;
    const int pos = pos0 + r;
    const int hi = a.causal ? min(pos, seq_len - 1) : seq_len - 1;      // last visible key
    const int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;       // first visible key
    const float sl2 = a.scale * 1.4426950408889634f;
    float m_used = -INFINITY, l = 0.0f;
    bool ok = true;
    for (int j = 0; j < nt; ++j) {
      ok = mbar_wait_warp(&s_full[h], j & 1, a.status, kKernelId, 0x640u + h, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, v[c]);
      tmem_ld_wait();
      // only tiles that touch the diagonal, the window's start or the end of the sequence need masks
      const int key0 = (t0 + j) * BKV;
      const bool need_mask = (key0 + BKV - 1 > (a.causal ? min(pos0, seq_len - 1) : seq_len - 1)) ||
                             (a.window > 0 && key0 < pos0 + BQ - a.window);
      if (need_mask) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int key = key0 + c * 32 + i;
            if (key > hi || key < lo) v[c][i] = 0xff800000u;            // -inf
          }
      }
      float mx[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mx[c] = __uint_as_float(v[c][0]);
#pragma unroll
        for (int i = 1; i < 32; ++i) mx[c] = fmaxf(mx[c], __uint_as_float(v[c][i]));
      }
      const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float alpha = 1.0f;
      if (mt > m_used && (m_used == -INFINITY || (mt - m_used) * sl2 > 8.0f)) {
        alpha = m_used == -INFINITY ? 0.0f : ex2_approx((m_used - mt) * sl2);
        m_used = mt;
      }
      const float mb = (m_used == -INFINITY ? 0.0f : m_used) * sl2;
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) {
        // (rare behind the first tiles; the scores stay in registers meanwhile)
#pragma unroll 1
        for (int c = 0; c < HD / 16; ++c) {
          uint32_t o[16];
          tmem_ld_32x16(o_addr + c * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x16(o_addr + c * 16, o);
        }
      }
      float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          // a masked score is -inf and its probability 0, also while no key of the row was visible
          const float p0 = ex2_approx(fmaf(__uint_as_float(v[c][i]), sl2, -mb));
          const float p1 = ex2_approx(fmaf(__uint_as_float(v[c][i + 1]), sl2, -mb));
          sum[c] += p0 + p1;
          pk[i >> 1] = pack_bf16x2(p0, p1);
        }
        tmem_st_32x16(s_addr + c * 16, pk);
      }
      l = l * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[h]);
    }
    if (ok) ok = mbar_wait_warp(&o_done[h], 0, a.status, kKernelId, 0x650u + h, abort_flag);
    if (ok) {
      tc_fence_after();
      float den = l;
      if (a.sink != nullptr)       // relative to the running maximum, like the row sum
        den += exp2f(fmaf(a.sink[head0 + h], 1.4426950408889634f, -m_used * sl2));
      const float inv = l > 0.0f ? 1.0f / den : 0.0f;
      const bool row_ok = r < rows;
      __nv_bfloat16* orow =
          a.out + static_cast<long long>(q_start + q0 + r) * a.ldo + (head0 + h) * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(o_addr + c * 32, o);
        tmem_ld_wait();
        if (!row_ok) continue;
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            w[e] = pack_bf16x2(__uint_as_float(o[i + 2 * e]) * inv,
                               __uint_as_float(o[i + 2 * e + 1]) * inv);
          *reinterpret_cast<uint4*>(orow + c * 32 + i) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      if (row_ok && a.lse != nullptr)
        a.lse[static_cast<long long>(head0 + h) * a.T + q_start + q0 + r] =
            l > 0.0f ? m_used * sl2 * 0.6931471805599453f + logf(l) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace fmha
}  // namespace b200
