// Prefill attention of two query tiles at once (included by attention_fmha.cu, whose Args and constants
// it uses), value dimension 128.  Two forms:
//   heads    head dimension 128, keys and values in the paged cache, query heads in pairs over one key head;
//            the tiles are 128 rows of two heads.  No soft cap, chunk or bias.
//   latent   latent attention over keys and values that were expanded per head into [keys, heads * 256] (128
//            columns of a key, 128 of a value), with 64 rotated key columns that all heads share; queries
//            have 192 columns; the tiles are 2 x 128 rows of one head.  Causal.  Off by default
//            (models/deepseek.py, USE_EXPANDED_PROMPTS).
//
// What bounds it: per 128 x 128 scores the tensor cores need 1024 cycles (Q K^T and P V; 1280 with 192
// columns) and the exponentials 1024 cycles of the special-function pipe, and one tile's chain scores ->
// softmax -> P V takes about 3500.  So two tiles are worked on, and their exponentials take turns: while one
// has the special-function pipe, the other's products, row maxima and hand-overs run.  (Left to themselves
// the two chains stay in step, with both at the special-function pipe and then both waiting for products:
// 8192 tokens of 32 heads 577 us, 2 x 2048 tokens 119, in turns 503 and 92; chains issued by one thread in
// a fixed order, without turns, 600 and 127.)  Every key tile is loaded once for both.
// Probabilities go back into the tensor memory that held the scores, from where P V takes them as its A
// operand: no shared-memory stores and no proxy fence in the chain.  P V of the first 64 keys starts when
// their probabilities are there.  One thread owns a row of 128 scores, read once into registers.
//
// Each tile's products are issued by a thread of its own (a wait and the issue of eight products take some
// 400 cycles, which one thread for both would put into both chains).  They execute in the order of issue, so
// the barrier that announces S(j) also says that P V(j - 1) has read its probabilities and finished its sums: the
// softmax warps may rescale the output in place without another wait.  The running maximum is raised only
// when it is exceeded by 8 in the log2 domain, as in the kernel for one head.
//
// One CTA per SM goes through pieces of work by falling number of keys, in rounds of the grid from either
// end: the longest first, and loads and first scores of the next piece run under the last products and
// the epilogue of the one before.  (A CTA for each piece, longest of a head first: 2 x 2048 tokens 17 per
// cent more time in set-ups and at the end of the grid.)
//
// Warps: 0 finds work and loads (lane = page and half of a key tile), 1 and 2 tcgen05.mma of the two tiles, 1
// owns tensor memory, 4..7 softmax and epilogue of the first tile, 8..11 of the second.
// Measured against the kernel that went before (one issuing thread, no turns, a CTA for each piece of work; the
// same bits from both), 32 heads, us: 8192 tokens 573 -> 488, 2 x 2048 tokens 113 -> 88, 7 x 1024 tokens 125 -> 104, 40
// requests of 40 tokens behind 100 71 -> 39.  Latent form, 2 x 1024 tokens of 128 heads with the expansion in front 206, where the absorbed form
// takes 826 with its products per head.
#pragma once

namespace b200 {
namespace fmha {

constexpr int kPairOffBar = 14 * kSub;            // behind query tiles and the ring of key and value units
constexpr int kPairThreads = 384;
constexpr int kPairSmemBytes = kPairOffBar + 512 + 1024;
constexpr uint32_t kPairColO = 256;               // scores of slot h: 128 h, outputs 256 + 128 h
static_assert(kPairSmemBytes <= 232448, "exceeds the shared memory of one CTA");

// two fp32 numbers in a 64-bit register, for the instructions that work on both
__device__ __forceinline__ uint64_t f2_pack(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t r, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(r));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// (three operands: half the instructions of a row maximum)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Tile of `rows` query rows number `rank` of the step by falling number of keys that it sees, by one warp.
// Tile i of a sequence has length c + i, with c the tiles of keys in front of the first one, so a sequence
// has at most one tile of each length.  Each lane keeps the sequence of its number in registers.
__device__ __forceinline__ void find_long_tile(const Args& a, int rows, int rank, int lane, int n_lane,
                                               int c_lane, int* seq, int* qt) {
  auto get = [&](int b, int* n, int* c) {
    if (b < 32) {
      *n = n_lane;
      *c = c_lane;
    } else {
      *n = *c = 0;
      if (b < a.B) {
        const int len = a.cu_q[b + 1] - a.cu_q[b];
        *n = (len + rows - 1) / rows;
        *c = max(0, a.seq_lens[b] - len) / rows;
      }
    }
  };
  auto count = [&](int t) {                     // tiles of length >= t
    int s = 0;
    for (int b = lane; b < a.B; b += 32) {
      int n, c;
      get(b, &n, &c);
      s += max(0, min(n, c + n - t));
    }
    return __reduce_add_sync(0xffffffffu, s);
  };
  int top = 0;
  for (int b = lane; b < a.B; b += 32) {
    int n, c;
    get(b, &n, &c);
    if (n > 0) top = max(top, c + n);
  }
  int lo = 0, hi = __reduce_max_sync(0xffffffffu, top);      // count(hi) = 0
  *seq = -1;
  *qt = 0;
  if (count(0) <= rank) return;
  while (hi - lo > 1) {                         // largest t with count(t) > rank
    const int mid = (lo + hi) >> 1;
    if (count(mid) > rank) lo = mid;
    else hi = mid;
  }
  int k = rank - count(lo + 1);                 // the k-th sequence with a tile of this length
  for (int b0 = 0; b0 < a.B; b0 += 32) {
    int n, c;
    get(b0 + lane, &n, &c);
    if (b0 + lane >= a.B) n = 0;
    const unsigned int vote = __ballot_sync(0xffffffffu, n > 0 && lo >= c && lo < c + n);
    const int here = __popc(vote);
    if (k < here) {
      const bool mine = (vote >> lane & 1u) != 0u && __popc(vote & ((1u << lane) - 1u)) == k;
      const int src = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
      *seq = b0 + src;
      *qt = lo - __shfl_sync(0xffffffffu, c, src);
      return;
    }
    k -= here;
  }
}

struct Work {            // what the TMA warp tells the others about a pair of tiles
  int seq;               // -1: no more work
  int row;               // first query row of the step
  int rows;              // valid rows of it (kLatent: of both slots)
  int pos;               // position of the first row
  int keys;              // of the sequence
  int head;              // head (kLatent) or first of two heads
  int t0;                // first key tile
  int nt[2];             // key tiles of both slots
  int pad[3];
};

template <bool kLatent>
__global__ void __launch_bounds__(kPairThreads, 1)
    fmha_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const Args a, const int total) {
  constexpr int HD = 128;                       // columns of a value
  constexpr int kQU = kLatent ? 3 : 2;          // units of 64 columns of a query or key
  constexpr int kUnits = 14 - 2 * kQU;          // ring
  constexpr int kTileUnits = kQU + 2;           // of a tile of keys and its values
  constexpr int RT = kLatent ? 2 * BQ : BQ;     // query rows of a piece of work
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* ring = smem + 2 * kQU * kSub;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kPairOffBar);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 1;
  uint64_t* w_full = bars + 2;              // [2] a Work is there
  uint64_t* w_empty = bars + 4;             // [2]
  uint64_t* s_full = bars + 6;              // per slot: scores are there
  uint64_t* p_half = bars + 8;              // per slot: output rescaled, half of the probabilities are there
  uint64_t* p_full = bars + 10;             // per slot: all probabilities
  uint64_t* o_done = bars + 12;             // per slot: the last product has finished
  uint64_t* turn = bars + 30;               // per slot: its exponentials of a tile are done
  uint64_t* k_full = bars + 14;             // [4] key tiles, tile t at t % 4
  uint64_t* k_empty = bars + 18;
  uint64_t* v_full = bars + 22;
  uint64_t* v_empty = bars + 26;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 32);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile Work* works = reinterpret_cast<volatile Work*>(tmem_slot + 2);
  static_assert(32 * 8 + 8 + 2 * sizeof(Work) <= 512, "barrier area");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 2);
    for (int i = 0; i < 4; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 2);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&w_full[i], 1);
      mbar_init(&w_empty[i], 10);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_half[i], 4);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1);
      mbar_init(&turn[i], 4);
    }
    *abort_flag = 0u;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  grid_release();
  grid_wait();

  // registers of the warps that compute: 2 x 200 and 96 of three warpgroups launched with 168 each
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    if (warp == 0) {
      // ---------------- work and TMA ----------------
      const int pairs = kLatent ? a.Hq : a.Hq >> 1;
      int n_lane = 0, c_lane = 0;
      if (lane < a.B) {
        const int len = a.cu_q[lane + 1] - a.cu_q[lane];
        n_lane = (len + RT - 1) / RT;
        c_lane = max(0, a.seq_lens[lane] - len) / RT;
      }
      int slot = 0, tile = 0;          // place in the ring, tiles so far
      for (int it = 0;; ++it) {
        // rounds of the grid in turn from either end, so that a CTA gets long and short tiles
        const int b = (it & 1) ? static_cast<int>(gridDim.x - 1 - blockIdx.x) : static_cast<int>(blockIdx.x);
        const int w = it * static_cast<int>(gridDim.x) + b;
        int seq = -1, qt = 0;
        if (w < total) find_long_tile(a, RT, w / pairs, lane, n_lane, c_lane, &seq, &qt);
        Work k = {};
        k.seq = seq;
        int q_start = 0, key_off = 0;
        if (seq >= 0) {
          q_start = a.cu_q[seq];
          const int q_len = a.cu_q[seq + 1] - q_start;
          k.keys = a.seq_lens[seq];
          k.row = q_start + qt * RT;
          k.rows = min(RT, q_len - qt * RT);
          k.pos = k.keys - q_len + qt * RT;
          k.head = kLatent ? w % pairs : 2 * (w % pairs);
          k.t0 = a.window > 0 ? max(0, k.pos - a.window + 1) / BKV : 0;
  #pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int off = kLatent ? h * BQ : 0;
            const int rows = min(BQ, k.rows - off);
            const int hi = a.causal ? min(k.keys, k.pos + off + rows) : k.keys;
            k.nt[h] = rows > 0 ? max(1, (hi + BKV - 1) / BKV - k.t0) : 0;
          }
          if constexpr (kLatent) {
            int s = 0;             // the sequences' keys follow each other, each from a whole tile on
            for (int i = lane; i < seq; i += 32) s += (a.seq_lens[i] + BKV - 1) / BKV * BKV;
            key_off = __reduce_add_sync(0xffffffffu, s);
          }
        }
        if (!mbar_wait_warp(&w_empty[it & 1], ((it >> 1) & 1) ^ 1, a.status, kKernelId, 0x600u, abort_flag))
          break;
        if (lane == 0) {
          volatile Work* o = works + (it & 1);
          o->seq = k.seq;
          if (seq >= 0) {
            o->row = k.row;
            o->rows = k.rows;
            o->pos = k.pos;
            o->keys = k.keys;
            o->head = k.head;
            o->t0 = k.t0;
            o->nt[0] = k.nt[0];
            o->nt[1] = k.nt[1];
          }
          mbar_arrive(&w_full[it & 1]);
        }
        __syncwarp();
        if (seq < 0) break;
        if (!mbar_wait_warp(q_empty, (it & 1) ^ 1, a.status, kKernelId, 0x602u, abort_flag)) break;
        if (lane == 0) {
          const int slots = k.nt[1] > 0 ? 2 : 1;
          mbar_expect_tx(q_full, slots * kQU * kSub);
          for (int h = 0; h < slots; ++h)
            for (int c = 0; c < kQU; ++c)
              tma_load_2d(smem + (h * kQU + c) * kSub, &tmQ, q_full,
                          (kLatent ? k.head : k.head + h) * (kQU * 64) + c * 64, k.row + (kLatent ? h * BQ : 0));
        }
        __syncwarp();
        const int nt = max(k.nt[0], k.nt[1]);
        bool ok = true;
        // entry of tile t in the ring: its last unit takes the place of unit `last - kUnits`, and entries are
        // given back in the order in which they came
        auto room = [&](int t, int last) {
          const int u = t * kTileUnits + last - kUnits;
          if (u >= 0) {
            const int told = u / kTileUnits;
            const bool key = u - told * kTileUnits < kQU;
            ok = mbar_wait_warp(key ? &k_empty[told & 3] : &v_empty[told & 3], (told >> 2) & 1, a.status, kKernelId,
                                0x610u + (told & 3), abort_flag);
          }
        };
        auto unit = [&](int u) {         // place of unit u of the entry that starts at `slot`
          const int s = slot + u;
          return ring + (s >= kUnits ? s - kUnits : s) * kSub;
        };
        auto next_units = [&](int n) {
          slot += n;
          if (slot >= kUnits) slot -= kUnits;
        };
        if constexpr (kLatent) {
          for (int j = 0; j < nt; ++j, ++tile) {
            const int y = key_off + j * BKV;
            room(tile, 2);
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(&k_full[tile & 3], 3 * kSub);
            __syncwarp();
            if (lane < 2) tma_load_2d(unit(lane), &tmK, &k_full[tile & 3], k.head * 256 + lane * 64, y);
            else if (lane == 2) tma_load_2d(unit(2), &tmV, &k_full[tile & 3], a.rope_col, y);
            next_units(3);
            room(tile, 4);
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(&v_full[tile & 3], 2 * kSub);
            __syncwarp();
            if (lane < 2) tma_load_2d(unit(lane), &tmK, &v_full[tile & 3], k.head * 256 + 128 + lane * 64, y);
            next_units(2);
          }
        } else {
          // lane = (page of 16 keys, half of the head dimension)
          const int kvh = k.head / (a.Hq / a.Hkv);
          const int* bt = a.block_tables + static_cast<long long>(seq) * a.max_blocks;
          const int last_tok = k.keys - 1;
          const int page = lane >> 1, half = lane & 1;
          auto row_of = [&](int j) {           // pages past the end: any valid page
            const int key = (k.t0 + j) * BKV + page * kPage;
            return lane < 2 * (BKV / kPage)
                       ? bt[min(key, last_tok) / a.block_size] * a.block_size + key % a.block_size
                       : 0;
          };
          int y = row_of(0);
          for (int j = 0; j < nt && ok; ++j, ++tile) {
            const int y_next = j + 1 < nt ? row_of(j + 1) : 0;
            for (int kv = 0; kv < 2; ++kv) {
              uint64_t* full = kv == 0 ? &k_full[tile & 3] : &v_full[tile & 3];
              room(tile, 1 + 2 * kv);
              if (!ok) break;
              if (lane == 0) mbar_expect_tx(full, kTile);
              __syncwarp();
              if (lane < 2 * (BKV / kPage))
                tma_load_2d(unit(half) + page * (kPage * 128), kv == 0 ? &tmK : &tmV, full, kvh * HD + half * 64, y);
              next_units(2);
            }
            y = y_next;
          }
        }
        if (!ok) break;
      }
    } else if (warp <= 2) {
      // ---------------- MMA issuers, one per slot ----------------
      if (elect_one()) {
        constexpr uint32_t kIdescS = make_idesc(BQ, BKV, 1, 1);
        constexpr uint32_t kIdescO = make_idesc(BQ, HD, 1, 1) | kIdescBMajorMN;
        constexpr uint32_t kIdescHalf = make_idesc(BQ, HD / 2, 1, 1) | kIdescBMajorMN;
        const int h = warp - 1;
        const uint32_t t_s = tmem + h * BKV, t_o = tmem + kPairColO + h * HD;
        const uint64_t q_desc = make_desc_k_sw128(smem_u32(smem) + h * kQU * kSub);
        const uint64_t k_desc = make_desc_k_sw128(smem_u32(ring));
        const uint64_t v_desc = make_desc_mn_sw128(smem_u32(ring), kSub);
        int slot = 0, tile = 0;
        uint32_t p_phase = 0;
        bool ok = true;
        auto issue_s = [&]() {
  #pragma unroll
          for (int u = 0; u < kQU; ++u) {
            int s = slot + u;
            if (kLatent && s >= kUnits) s -= kUnits;
            const uint64_t kd = k_desc + static_cast<uint32_t>(s * (kSub >> 4));
  #pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_f16(t_s, q_desc + static_cast<uint32_t>(u * (kSub >> 4) + ks * 2), kd + static_cast<uint32_t>(ks * 2),
                       kIdescS, u > 0 || ks > 0 ? 1u : 0u);
          }
          umma_commit(&s_full[h]);
        };
        auto next_units = [&](int n) {
          slot += n;
          if (slot >= kUnits) slot -= kUnits;
        };
        auto wait_tile = [&](uint64_t* full, int t) {
          ok = ok && mbar_wait(&full[t & 3], (t >> 2) & 1, a.status, kKernelId, 0x620u + (t & 3), abort_flag);
          tc_fence_after();
        };
        for (int it = 0;; ++it) {
          ok = mbar_wait(&w_full[it & 1], (it >> 1) & 1, a.status, kKernelId, 0x630u, abort_flag);
          if (!ok) break;
          const int seq = works[it & 1].seq;
          const int nt = works[it & 1].nt[h], n = max(nt, works[it & 1].nt[h ^ 1]);
          mbar_arrive(&w_empty[it & 1]);
          if (seq < 0) break;
          ok = mbar_wait(q_full, it & 1, a.status, kKernelId, 0x631u, abort_flag);
          wait_tile(k_full, tile);
          if (!ok) break;
          // (a slot without rows, or one that sees fewer keys than the other, gives tiles back all the same,
          // once they are there: else it could run ahead of the other by a round of the barrier)
          if (nt > 0) {
            issue_s();
            umma_commit(&k_empty[tile & 3]);
            if (n == 1) umma_commit(q_empty);
          } else {
            mbar_arrive(&k_empty[tile & 3]);
            if (n == 1) mbar_arrive(q_empty);
          }
          next_units(kQU);
          for (int j = 0; j < n; ++j, ++tile) {
            wait_tile(v_full, tile);
            if (!ok) break;
            if (j < nt) {
              const uint64_t vd = v_desc + static_cast<uint32_t>(slot * (kSub >> 4));
  #pragma unroll
              for (int part = 0; part < 2; ++part) {
                ok = mbar_wait(part == 0 ? &p_half[h] : &p_full[h], p_phase, a.status, kKernelId, 0x632u + h,
                               abort_flag);
                if (!ok) break;
                tc_fence_after();
                if (!kLatent || slot + 1 < kUnits) {
  #pragma unroll
                  for (int ks = 0; ks < 4; ++ks) {
                    const int step = part * 4 + ks;
                    umma_f16_ts(t_o, t_s + step * 8, vd + static_cast<uint32_t>(step * (2048 >> 4)), kIdescO,
                                (j > 0 || part > 0 || ks > 0) ? 1u : 0u);
                  }
                } else {         // the two units of the tile lie at the ring's end and start
                  for (int c = 0; c < 2; ++c) {
                    const uint64_t half = c == 0 ? vd : v_desc;
  #pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                      const int step = part * 4 + ks;
                      umma_f16_ts(t_o + c * 64, t_s + step * 8, half + static_cast<uint32_t>(step * (2048 >> 4)),
                                  kIdescHalf, (j > 0 || part > 0 || ks > 0) ? 1u : 0u);
                    }
                  }
                }
              }
              if (!ok) break;
              p_phase ^= 1u;
              if (j + 1 == nt) umma_commit(&o_done[h]);
              umma_commit(&v_empty[tile & 3]);
            } else {
              mbar_arrive(&v_empty[tile & 3]);
            }
            next_units(2);
            if (j + 1 < n) {
              wait_tile(k_full, tile + 1);
              if (!ok) break;
              if (j + 1 < nt) {
                issue_s();
                umma_commit(&k_empty[(tile + 1) & 3]);
                if (j + 2 == n) umma_commit(q_empty);
              } else {
                mbar_arrive(&k_empty[(tile + 1) & 3]);
                if (j + 2 == n) mbar_arrive(q_empty);
              }
              next_units(kQU);
            }
          }
          if (!ok) break;
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    // ---------------- softmax + epilogue: one thread per query row ----------------
    const int h = (warp - 4) >> 2;
    const int qd = warp & 3;                    // TMEM lane quarter
    const int r = qd * 32 + lane;               // query row in the tile
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(qd * 32) << 16);
    const uint32_t s_addr = lane_addr + h * BKV, o_addr = lane_addr + kPairColO + h * HD;
    const float sl2 = a.scale * 1.4426950408889634f;
    const uint64_t sl2_2 = f2_pack(sl2, sl2);
    uint32_t s_phase = 0, o_phase = 0, t_phase = 0;
    // Turns: key tiles that both slots have, one after the other over all pieces of work: slot 0, slot 1, slot 0 ...
    // Each slot waits for the other's turn before every one of them (the very first excepted), also across
    // pieces: a slot that went on without could complete the next turn before a warp of the other has looked at this
    // one, and that warp would wait for a parity that has come back.
    int both_before = 0;                        // such tiles in the pieces so far
    for (int it = 0;; ++it) {
      if (!mbar_wait_warp(&w_full[it & 1], (it >> 1) & 1, a.status, kKernelId, 0x640u, abort_flag)) break;
      const volatile Work* k = works + (it & 1);
      const int seq = k->seq;
      const int nt = k->nt[h], nt_both = min(nt, k->nt[h ^ 1]), t0 = k->t0, keys = k->keys, head = kLatent ? k->head : k->head + h;
      const int pos0 = k->pos + (kLatent ? h * BQ : 0), row0 = k->row + (kLatent ? h * BQ : 0);
      const int rows = k->rows - (kLatent ? h * BQ : 0);
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_empty[it & 1]);
      if (seq < 0) break;
      if (nt == 0) continue;
      const int pos = pos0 + r;
      const int hi = a.causal ? min(pos, keys - 1) : keys - 1;          // last visible key
      const int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;     // first visible key
      // keys that all rows of the tile see, and that all rows of the warp see
      const int edge = a.causal ? min(pos0, keys - 1) : keys - 1;
      const int hi_warp = a.causal ? min(pos0 + qd * 32, keys - 1) : keys - 1;
      const int lo_warp = pos0 + qd * 32 + 31 - a.window + 1;
      float m_used = -INFINITY, l = 0.0f;
      bool ok = true;
      for (int j = 0; j < nt; ++j) {
        ok = mbar_wait_warp(&s_full[h], s_phase, a.status, kKernelId, 0x641u + h, abort_flag);
        if (!ok) break;
        s_phase ^= 1u;
        tc_fence_after();
        uint32_t v[4][32];
        const int key0 = (t0 + j) * BKV;
        const bool need_mask = (key0 + BKV - 1 > edge) || (a.window > 0 && key0 < pos0 + BQ - a.window);
        float mx[4];
        auto masked = [&](int c) {          // chunk of 32 keys, where a row of the warp does not see all of them
          const int first = key0 + c * 32;
          if (need_mask && (first + 31 > hi_warp || (a.window > 0 && first < lo_warp))) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i > hi - first || i < lo - first) v[c][i] = 0xff800000u;            // -inf
          }
        };
        auto row_max = [&](int c) {
          float m0 = fmaxf(__uint_as_float(v[c][0]), __uint_as_float(v[c][1]));
          float m1 = fmaxf(__uint_as_float(v[c][2]), __uint_as_float(v[c][3]));
#pragma unroll
          for (int i = 4; i < 32; i += 4) {
            m0 = max3(m0, __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
            m1 = max3(m1, __uint_as_float(v[c][i + 2]), __uint_as_float(v[c][i + 3]));
          }
          mx[c] = fmaxf(m0, m1);
        };
        tmem_ld_32x32(s_addr, v[0]);
        tmem_ld_32x32(s_addr + 32, v[1]);
        tmem_ld_wait();
        tmem_ld_32x32(s_addr + 64, v[2]);
        tmem_ld_32x32(s_addr + 96, v[3]);
        masked(0);
        masked(1);
        row_max(0);
        row_max(1);
        tmem_ld_wait();
        masked(2);
        masked(3);
        row_max(2);
        row_max(3);
        const float mt = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
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
        const uint64_t mb2 = f2_pack(-mb, -mb);
        if (j < nt_both && both_before + j + h > 0) {
          mbar_pass_warp(&turn[h ^ 1], t_phase, a.status, kKernelId, 0x644u + h, abort_flag);
          t_phase ^= 1u;
        }
        float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};      // of 32 keys each
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            // a masked score is -inf and its probability 0, also while no key of the row was visible
            const uint64_t x = f2_fma(f2_pack(__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])),
                                      sl2_2, mb2);
            float p0, p1;
            f2_unpack(x, p0, p1);
            p0 = ex2_approx(p0);
            p1 = ex2_approx(p1);
            sum[c] += p0 + p1;
            pk[i >> 1] = pack_bf16x2(p0, p1);
          }
          if (c == 3 && lane == 0 && j < nt_both) mbar_arrive(&turn[h]);
          tmem_st_32x16(s_addr + c * 16, pk);
          if (c == 1) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_half[h]);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[h]);
        l = l * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      }
      both_before += nt_both;
      if (ok) ok = mbar_wait_warp(&o_done[h], o_phase, a.status, kKernelId, 0x650u + h, abort_flag);
      if (!ok) break;
      o_phase ^= 1u;
      tc_fence_after();
      float den = l;
      if (a.sink != nullptr)       // relative to the running maximum, like the row sum
        den += exp2f(fmaf(a.sink[head], 1.4426950408889634f, -m_used * sl2));
      const float inv = l > 0.0f ? 1.0f / den : 0.0f;
      const bool row_ok = r < rows;
      __nv_bfloat16* orow = a.out + static_cast<long long>(row0 + r) * a.ldo + head * HD;
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
        a.lse[static_cast<long long>(head) * a.T + row0 + r] =
            l > 0.0f ? m_used * sl2 * 0.6931471805599453f + logf(l) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace fmha
}  // namespace b200
