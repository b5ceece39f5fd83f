// Paged prefill on pairs of CTAs (tcgen05 cta_group::2), for query blocks of more than one 128-row tile.
//
// What bounds a one-CTA tile of 128 query rows is the K/V traffic from L2: at head_dim 256 every
// 64-key tile brings 64 KB into each SM for 1536 cycles of tensor work, and about 21 bytes per clock
// arrive per SM (3100 cycles).  Here the two CTAs of a cluster own the two halves of a 256-row query
// tile and share every K/V tile: an MMA of the pair (M 256 = 128 rows per CTA) reads half of its B
// operand from each CTA's shared memory, so each loads half of the keys of a K tile and half of the
// columns of a V tile, i.e. half the bytes per row.
//
//   S[j] = Q K_j^T    M 256, N 128 keys: CTA r holds keys [64 r, 64 r + 64) of the K tile
//   O   += P[j] V_j   M 256, N head_dim: CTA r holds columns [r head_dim / 2, ...) of the V tile
//
// The MMAs are issued by the leader (rank 0) and fill both CTAs' tensor memory; a commit signals both.
// S has two buffers and runs two key tiles ahead of PV, so the softmax warps never wait for the tensor
// pipe.  TMEM columns: S[b] at 128 b, O at 256.
//
//   warps 0-3   softmax: thread r owns row r of this CTA's half (TMEM lane r)
//   warp 4      MMA issuer (leader)
//   warp 5      relay: a buffer that is full here is announced to the leader, behind the proxy fence
//               that its generic-proxy copies (ragged pages, per-token rows) need
//   warps 6 ..  producers: one warp issues TMA boxes (PAGED), ten gather per-token rows
//
// Tile layouts are those of prefill_tc.cuh (128-byte swizzle; K tile [head_dim/64][64 rows][128 B],
// V tile [head_dim/128][128 rows][128 B], Q tile [head_dim/64][128 rows][128 B]).  Every wait is bounded.
#pragma once

#include "prefill_tc.cuh"

namespace msgl {

template <int HD, bool PAGED>
struct PairShape {
  static constexpr int kRows = 128;                       // query rows of a CTA
  static constexpr int kBM = 256;                         // of the pair
  static constexpr int kBN = 128;                         // keys of a tile
  static constexpr int kQBytes = kRows * HD * 2;
  static constexpr int kBufBytes = kBN * HD;              // half a K (or V) tile
  static constexpr int kBufs = 128 * 1024 / kBufBytes;    // 4 at head_dim 256, 8 at 128
  static constexpr int kSmemBytes = kQBytes + kBufs * kBufBytes + 1024;
  static constexpr int kMmaWarp = 4, kRelayWarp = 5, kProducerWarp0 = 6;
  static constexpr int kWarps = PAGED ? 8 : 16;
  static constexpr int kThreads = kWarps * 32;
  static constexpr int kOCol = 2 * kBN;
};

// ---------------------------------------------------------------- cluster and cta_group::2 wrappers
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on the barrier at this address in CTA `rank` of the cluster.
__device__ __forceinline__ void mbar_arrive_at(uint32_t bar, uint32_t rank) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [ra];\n\t}" ::"r"(bar),
      "r"(rank)
      : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
// Bounded, warp-uniform wait for arrivals from either CTA (see mbar_wait_limit).
__device__ __forceinline__ bool mbar_wait_warp_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  bool ok = mbar_try_wait_cluster(bar, parity) != 0;
  if (!ok) {
    const long long t0 = clock64();
    while (true) {
      ok = mbar_try_wait_cluster(bar, parity) != 0;
      if (ok) break;
      if (*abort_flag != 0 || clock64() - t0 > kTcWaitCycles) {
        *abort_flag = 1;
        break;
      }
    }
  }
  return __all_sync(0xffffffffu, ok ? 1 : 0) != 0;
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// The MMAs issued so far, when done, arrive on the barrier at this address in both CTAs.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .b16 m;\n\tmov.b16 m, 3;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_mma_pair_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_mma_pair_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Instruction descriptor as idesc_m128, M = 256.
template <typename T>
__device__ __forceinline__ uint32_t idesc_m256(uint32_t n, uint32_t b_mn) {
  return (idesc_m128<T>(n, b_mn) & ~(0x1fu << 24)) | ((256u >> 4) << 24);
}

struct PairBarriers {
  uint64_t q_full, q_pair;               // Q of this CTA / of both (leader)
  uint64_t full[8], pair_full[8], empty[8];
  uint64_t s_full[2], p_full[2], pv_done[2];
  uint64_t idx_sync;                     // per-token form: the producers' own barrier
};

template <typename T, int HD, bool PAGED>
__global__ void __launch_bounds__(PairShape<HD, PAGED>::kThreads, 1)
    prefill_pair_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap tm_k,
                        const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_q) {
  using Shape = PairShape<HD, PAGED>;
  constexpr int BM = Shape::kBM, BN = Shape::kBN, ROWS = Shape::kRows, NB = Shape::kBufs;
  constexpr int KEYS = BN / 2;                  // keys of a K tile in this CTA
  constexpr int CH = HD / 8;                    // 16-byte chunks of a token row
  constexpr int VCH = CH / 2;                   // ... of its half of a V row
  constexpr int NPROD = (Shape::kWarps - Shape::kProducerWarp0) * 32;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ PairBarriers bars;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ int s_slots[PAGED ? 1 : 3 * BN];   // slot ids of the key tiles being copied / next to copy

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int G = p.group;
  const int rank = static_cast<int>(cluster_rank());
  const bool q_tma = PAGED && p.q_tma != 0;

  auto bar_full = [&](int bf) { return smem_u32(&bars.full[bf]); };
  auto bar_pair = [&](int bf) { return smem_u32(&bars.pair_full[bf]); };
  auto bar_empty = [&](int bf) { return smem_u32(&bars.empty[bf]); };
  auto bar_s = [&](int b) { return smem_u32(&bars.s_full[b]); };
  auto bar_p = [&](int b) { return smem_u32(&bars.p_full[b]); };
  auto bar_pv = [&](int b) { return smem_u32(&bars.pv_done[b]); };
  const uint32_t bar_q = smem_u32(&bars.q_full), bar_qp = smem_u32(&bars.q_pair);

  if (tid == 0) {
    s_abort = 0;
    mbar_init(bar_q, q_tma ? 1 : Shape::kThreads);
    mbar_init(bar_qp, 2);
    mbar_init(smem_u32(&bars.idx_sync), NPROD);
    for (int bf = 0; bf < NB; ++bf) {
      mbar_init(bar_full(bf), PAGED ? (NPROD / 32) * 33 : NPROD);   // (33: see prefill_tc.cuh)
      mbar_init(bar_pair(bf), 2);
      mbar_init(bar_empty(bf), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_s(b), 1);
      mbar_init(bar_p(b), 2 * (ROWS / 32));
      mbar_init(bar_pv(b), 1);
    }
    fence_mbar_init();
  }
  if (warp == Shape::kMmaWarp) {
    tmem_alloc_pair(smem_u32(&s_tmem_base), 512);
    tmem_relinquish_pair();
  }
  if (!p.early) grid_dependency_wait();
  ItemCoord it;
  const bool have_item = find_item<Shape::kThreads>(p, static_cast<int>(blockIdx.x) / 2, BM,
                                                    reinterpret_cast<int*>(smem_raw), it);
  if (p.early) grid_dependency_wait();
  grid_dependency_launch();
  tc_fence_before();
  cluster_sync_all();           // the barriers of both CTAs exist (and the CTA's own set-up is done)
  tc_fence_after();
  const uint32_t tmem = s_tmem_base;
  if (!have_item) {             // the same in both CTAs: a launch rank past the last item
    if (warp == Shape::kMmaWarp) tmem_dealloc_pair(tmem, 512);
    return;
  }
  const int h = it.h;
  const SeqShape sq = load_seq_shape(p, it.b, BM);
  if (PAGED && it.first && rank == 0 && tid == 0 && p.status) {
    // a length that is negative or exceeds the sequence's pages was clamped: report it
    const int64_t cap = static_cast<int64_t>(p.page_indptr[it.b + 1] - p.page_indptr[it.b]) * p.page_size;
    const int len = p.kv_lens[it.b];
    if (len < 0 || len > cap) atomicExch(p.status, 2);
  }

  // ---- geometry: the pair's key range, this CTA's rows
  const int pk0 = it.qt * BM;
  const int rows_pair = min(BM, sq.tq * G - pk0);                       // >= 1
  const int rows_valid = max(0, min(ROWS, rows_pair - rank * ROWS));
  const int tok_first = pk0 / G;
  const int tok_last = (pk0 + rows_pair - 1) / G;
  int kv_lo = p.window > 0 ? max(0, sq.prefix + tok_first - p.window + 1) : 0;
  kv_lo = (kv_lo / BN) * BN;
  const int kv_hi = p.is_cross ? sq.L : min(sq.L, sq.prefix + tok_last + 1);   // keys from here on are never read
  const int ntiles = kv_hi > kv_lo ? ceil_div(kv_hi - kv_lo, BN) : 0;

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem0;
  const uint32_t ring = smem0 + Shape::kQBytes;
  volatile int* abort_flag = &s_abort;

  // ---- Q: TMA boxes where a box holds whole tokens (128 rows divide by the group), else 16-byte
  // copies by all threads (by the two producer warps alone they took 24000 cycles at head_dim 256)
  if (q_tma) {
    // (rows past the sequence's last query token hold a neighbour's rows: computed on, never written)
    if (warp == Shape::kProducerWarp0 && elect_one()) {
      prefetch_tensormap(&tm_q);
      mbar_arrive_expect_tx(bar_q, Shape::kQBytes);
#pragma unroll
      for (int c = 0; c < HD / 64; ++c)
        tma_load_3d(q_smem + c * (ROWS * 128), &tm_q, c * 64, h * G, sq.q_begin + tok_first + rank * (ROWS / G), bar_q);
    }
    __syncwarp();
  } else {
    const T* q = static_cast<const T*>(p.q);
    const int chunk = tid % CH;
    for (int row = tid / CH; row < ROWS; row += Shape::kThreads / CH) {
      const int pk = pk0 + rank * ROWS + row;
      const int tl = pk / G, g = pk - tl * G;
      const bool ok = row < rows_valid;
      const int64_t off =
          ok ? ((static_cast<int64_t>(sq.q_begin + tl) * p.hq + static_cast<int64_t>(h) * G + g) * HD) : 0;
      cp_async_16(q_smem + tc_tile_offset<ROWS>(row, chunk),
                  reinterpret_cast<const unsigned char*>(q + off) + chunk * 16, ok ? 16 : 0);
    }
    cp_async_mbar_arrive(bar_q);
  }
  // the gate's rows on their way into L2: the epilogue wants them
  if (p.gate && warp == Shape::kRelayWarp) {
    for (int e = lane; e < rows_valid * (HD / 64); e += 32) {
      const int pk = pk0 + rank * ROWS + e / (HD / 64);
      const int tl = pk / G, g = pk - tl * G;
      prefetch_l2(static_cast<const T*>(p.gate) +
                  (static_cast<int64_t>(sq.q_begin + tl) * p.hq + static_cast<int64_t>(h) * G + g) * HD +
                  e % (HD / 64) * 64);
    }
  }

  if (warp >= Shape::kMmaWarp) {
    if constexpr (!PAGED) reg_dec<88>();
    if (warp >= Shape::kProducerWarp0) {
      // =========================================================== producers
      const int ptid = tid - Shape::kProducerWarp0 * 32;
      const unsigned char* kbase = static_cast<const unsigned char*>(p.k_cache);
      const unsigned char* vbase = static_cast<const unsigned char*>(p.v_cache);
      const int64_t slot_stride = static_cast<int64_t>(p.hkv) * (HD * 2);
      const int64_t head_off = static_cast<int64_t>(h) * (HD * 2);
      const int64_t v_off = head_off + rank * HD;          // this CTA's half of the V columns, bytes
      bool alive = true;
      if constexpr (PAGED) {
        {
          // (the boxes of a tile are dealt to both producer warps: one alone issues 31 B/clk)
          constexpr int NPW = NPROD / 32;
          const int pw = warp - Shape::kProducerWarp0;
          constexpr int PPT = BN / kTmaBoxRows;            // 8 pages of a tile, a lane each
          constexpr uint32_t kBoxBytes = kTmaBoxRows * 128;
          const int32_t* pages = p.page_indices + sq.kv_begin;
          if (lane == 0) {
            prefetch_tensormap(&tm_k);
            prefetch_tensormap(&tm_v);
          }
          // y = first pool row of the lane's page, n = rows of it that belong to the sequence
          auto fetch_box = [&](int tile, int& y, int& n) {
            y = 0;
            n = 0;
            const int t0 = kv_lo + tile * BN + lane * kTmaBoxRows;
            if (lane < PPT && tile < ntiles && t0 < kv_hi) {
              const int pg = __ldg(pages + t0 / p.page_size);
              const int64_t row0 = static_cast<int64_t>(pg) * p.page_size + t0 % p.page_size;
              const int nv = min(kTmaBoxRows, sq.L - t0);
              if (pg < 0 || row0 + nv > p.num_slots) {
                if (p.status) atomicExch(p.status, 2);     // page outside the pool: rows read as zeros
              } else {
                y = static_cast<int>(row0);
                n = nv;
              }
            }
          };
          int issued_seq = -1;
          auto produce = [&](int seq, bool is_k, int y, int n) {
            const int bf = seq % NB;
            alive = mbar_wait_warp(bar_empty(bf), ((seq / NB) & 1) ^ 1, abort_flag);
            if (!alive) return;
            const uint32_t dst = ring + bf * Shape::kBufBytes;
            const uint32_t bar = bar_full(bf);
            // K: this CTA's half of the pages, all columns; V: all pages, its half of the columns
            const uint32_t full_mask = __ballot_sync(0xffffffffu, n == kTmaBoxRows);
            const int page0 = is_k ? rank * (PPT / 2) : 0, npages = is_k ? PPT / 2 : PPT;
            const uint32_t mine = ((1u << npages) - 1u) << page0;
            uint32_t rest = mine & ~full_mask;
            constexpr int MINE = (PPT / 2) * (HD / 64) / NPW;   // boxes of a warp
            int yk[MINE], boxes = 0;
#pragma unroll
            for (int k = 0; k < MINE; ++k) {
              const int i = page0 + (pw + k * NPW) % npages;
              yk[k] = __shfl_sync(0xffffffffu, y, i);
              if (((full_mask >> i) & 1u) == 0) yk[k] = -1;
              boxes += yk[k] >= 0 ? 1 : 0;
            }
            const uint32_t block_bytes = (is_k ? KEYS : BN) * 128;
            if (elect_one()) {
              const CUtensorMap* tm = is_k ? &tm_k : &tm_v;
              const int x0 = h * HD + (is_k ? 0 : rank * (HD / 2));
              mbar_arrive_expect_tx(bar, boxes * kBoxBytes);
#pragma unroll
              for (int k = 0; k < MINE; ++k) {
                const int id = pw + k * NPW;
                if (yk[k] >= 0)
                  tma_load_2d(dst + (id / npages) * block_bytes + (id % npages) * kBoxBytes, tm,
                              x0 + (id / npages) * 64, yk[k], bar);
              }
              if (rest == 0) mbar_arrive_n(bar, 32);     // (else the lanes arrive behind their own copies)
            }
            __syncwarp();
            const bool ragged = rest != 0;
            const unsigned char* src = is_k ? kbase + head_off : vbase + v_off;
            const int ch = is_k ? CH : VCH;
            while (rest) {   // warp-uniform: ragged or out-of-range pages, row by row, zeros behind the end
              const int i = __ffs(rest) - 1;
              rest &= rest - 1;
              if (i % NPW != pw) continue;
              const int yi = __shfl_sync(0xffffffffu, y, i), ni = __shfl_sync(0xffffffffu, n, i);
              const int row_i = (i - page0) * kTmaBoxRows;
              for (int e = lane; e < kTmaBoxRows * ch; e += 32) {
                const int row = e / ch, chunk = e % ch;
                const bool ok = row < ni;
                const int64_t off = (ok ? static_cast<int64_t>(yi + row) * slot_stride : 0) + chunk * 16;
                const uint32_t so = is_k ? tc_tile_offset<KEYS>(row_i + row, chunk) : tc_tile_offset<BN>(row_i + row, chunk);
                cp_async_16(dst + so, src + off, ok ? 16 : 0);
              }
            }
            if (ragged) cp_async_mbar_arrive(bar);
            issued_seq = seq;
          };
          int wy[3], wn[3];
#pragma unroll
          for (int t = 0; t < 3; ++t) fetch_box(t, wy[t], wn[t]);
#pragma unroll 1
          for (int j = -2; j < ntiles && alive; ++j) {     // K two tiles ahead of V
            int ny = 0, nn = 0;
            if (j >= 0) {
              fetch_box(j + 3, ny, nn);                     // in flight while this step's copies are issued
              produce(ring_seq_v<2>(j), false, wy[0], wn[0]);
              if (!alive) break;
            }
            if (j + 2 < ntiles) {
              const int k = j < 0 ? j + 2 : 2;
              produce(ring_seq_k<2>(j + 2), true, k == 0 ? wy[0] : k == 1 ? wy[1] : wy[2],
                      k == 0 ? wn[0] : k == 1 ? wn[1] : wn[2]);
            }
            if (j >= 0) {
              wy[0] = wy[1];
              wn[0] = wn[1];
              wy[1] = wy[2];
              wn[1] = wn[2];
              wy[2] = ny;
              wn[2] = nn;
            }
          }
          if (!alive) {
            // gave up: let the bulk copies still in flight land before the shared memory goes away; bounded
            const long long t0 = clock64();
            for (int i = max(0, issued_seq - NB + 1); i <= issued_seq; ++i) {
              while (!mbar_try_wait(bar_full(i % NB), (i / NB) & 1) && clock64() - t0 < 2000000LL) {
              }
            }
          }
        }
      } else {
        // slot ids of a tile: one coalesced load, two tiles ahead of their use, staged in shared memory
        const int32_t* idx = p.kv_indices + sq.kv_begin;
        auto fetch_slot = [&](int tile) -> int {
          const int t = kv_lo + tile * BN + ptid;
          return (ptid < BN && tile < ntiles && t < kv_hi) ? __ldg(idx + t) : -1;
        };
        auto stage_slot = [&](int tile, int slot) {
          if (ptid < BN) {
            if (slot < -1 || static_cast<int64_t>(slot) >= p.num_slots) {
              if (p.status) atomicExch(p.status, 2);
              slot = -1;
            }
            s_slots[(tile % 3) * BN + ptid] = slot;
          }
        };
        uint32_t idx_phase = 0;
        const uint32_t bar_idx = smem_u32(&bars.idx_sync);
        auto producers_sync = [&]() {
          mbar_arrive(bar_idx);
          alive = mbar_wait_warp(bar_idx, idx_phase, abort_flag);
          idx_phase ^= 1;
        };
        auto produce = [&](int seq, bool is_k, int tile) {
          const int bf = seq % NB;
          alive = mbar_wait_warp(bar_empty(bf), ((seq / NB) & 1) ^ 1, abort_flag);
          if (!alive) return;
          const uint32_t dst = ring + bf * Shape::kBufBytes;
          const int* slots = s_slots + (tile % 3) * BN;
          if (is_k) {
            for (int e = ptid; e < KEYS * CH; e += NPROD) {
              const int row = e / CH, chunk = e % CH;
              const int slot = slots[rank * KEYS + row];
              const int64_t off = (slot >= 0 ? static_cast<int64_t>(slot) * slot_stride + head_off : 0) + chunk * 16;
              cp_async_16(dst + tc_tile_offset<KEYS>(row, chunk), kbase + off, slot >= 0 ? 16 : 0);
            }
          } else {
            for (int e = ptid; e < BN * VCH; e += NPROD) {
              const int row = e / VCH, chunk = e % VCH;
              const int slot = slots[row];
              const int64_t off = (slot >= 0 ? static_cast<int64_t>(slot) * slot_stride + v_off : 0) + chunk * 16;
              cp_async_16(dst + tc_tile_offset<BN>(row, chunk), vbase + off, slot >= 0 ? 16 : 0);
            }
          }
          cp_async_mbar_arrive(bar_full(bf));
        };
        for (int t = 0; t < 3; ++t) stage_slot(t, fetch_slot(t));
        producers_sync();
#pragma unroll 1
        for (int j = -2; j < ntiles && alive; ++j) {
          const int next_slot = j >= 0 ? fetch_slot(j + 3) : -1;
          if (j >= 0) produce(ring_seq_v<2>(j), false, j);
          if (alive && j + 2 < ntiles) produce(ring_seq_k<2>(j + 2), true, j + 2);
          if (!alive) break;
          if (j >= 0) {
            producers_sync();                   // every producer is done reading tile j's ids
            if (!alive) break;
            stage_slot(j + 3, next_slot);       // takes tile j's place
            producers_sync();
          }
        }
      }
      cp_async_wait<0>();
      if (!alive && p.status && ptid == 0) atomicExch(p.status, 1);
    } else if (warp == Shape::kRelayWarp) {
      // =========================================================== relay
      bool alive = true;
      if (ntiles > 0) {
        alive = mbar_wait_warp(bar_q, 0, abort_flag);
        if (alive) {
          fence_proxy_async_smem();
          if (lane == 0) mbar_arrive_at(bar_qp, 0);
        }
      }
      auto announce = [&](int seq) {
        const int bf = seq % NB;
        alive = mbar_wait_warp(bar_full(bf), (seq / NB) & 1, abort_flag);
        if (!alive) return;
        fence_proxy_async_smem();
        if (lane == 0) mbar_arrive_at(bar_pair(bf), 0);
      };
#pragma unroll 1
      for (int j = -2; j < ntiles && alive; ++j) {
        if (j >= 0) announce(ring_seq_v<2>(j));
        if (alive && j + 2 < ntiles) announce(ring_seq_k<2>(j + 2));
      }
      if (!alive && p.status && lane == 0) atomicExch(p.status, 1);
    } else if (warp == Shape::kMmaWarp && rank == 0) {
      // =========================================================== MMA issuer
      const uint32_t idesc_s = idesc_m256<T>(BN, 0);
      const uint32_t idesc_pv = idesc_m256<T>(HD, 1);
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t desc_k = smem_desc_sw128(0, 16, 1024);                 // Q / K: K-major
      const uint64_t desc_v = smem_desc_sw128(0, BN * 128, 1024);           // V: MN-major
      const int last_seq = ring_seq_v<2>(ntiles - 1);
      bool alive = true;
      auto acquire = [&](int seq) {
        alive = mbar_wait_warp_cluster(bar_pair(seq % NB), (seq / NB) & 1, abort_flag);
        if (alive) tc_fence_after();
      };
      // frees a ring buffer in both CTAs (only while somebody will fill it again)
      auto release = [&](int seq) {
        if (seq + NB <= last_seq) tc_commit_pair(bar_empty(seq % NB));
      };
      if (ntiles > 0) alive = mbar_wait_warp_cluster(bar_qp, 0, abort_flag);
#pragma unroll 1
      for (int j = -2; j < ntiles && alive; ++j) {
        const bool do_pv = j >= 0, do_s = j + 2 < ntiles;
        const int sv = ring_seq_v<2>(j), sk = ring_seq_k<2>(j + 2);
        if (do_pv) acquire(sv);
        if (alive && do_s) acquire(sk);
        if (alive && do_pv) {
          alive = mbar_wait_warp_cluster(bar_p(j & 1), (j >> 1) & 1, abort_flag);
          tc_fence_after();
        }
        if (!alive) break;
        const uint32_t vb = (ring + (do_pv ? sv % NB : 0) * Shape::kBufBytes) >> 4;
        const uint32_t kb = (ring + (do_s ? sk % NB : 0) * Shape::kBufBytes) >> 4;
        const uint32_t qa = q_smem >> 4;
        const uint32_t o_tm = tmem_u + Shape::kOCol;
        const uint32_t ps_tm = tmem_u + (j & 1) * BN;       // P of tile j, then S of tile j + 2
        if (elect_one()) {
          if (do_pv) {
#pragma unroll
            for (int ks = 0; ks < BN / 16; ++ks)
              tc_mma_pair_ts(o_tm, ps_tm + ks * 8, desc_v | (vb + ks * (2048 >> 4)), idesc_pv,
                             (j == 0 && ks == 0) ? 0u : 1u);
            tc_commit_pair(bar_pv(j & 1));
            release(sv);
          }
          if (do_s) {
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
              const uint32_t qoff = ((ks >> 2) * (ROWS * 128) + (ks & 3) * 32) >> 4;
              const uint32_t koff = ((ks >> 2) * (KEYS * 128) + (ks & 3) * 32) >> 4;
              tc_mma_pair_ss(ps_tm, desc_k | (qa + qoff), desc_k | (kb + koff), idesc_s, ks > 0 ? 1u : 0u);
            }
            tc_commit_pair(bar_s(j & 1));
            release(sk);
          }
        }
        __syncwarp();
      }
      if (!alive && p.status && lane == 0) atomicExch(p.status, 1);
    }
  } else {
    // =========================================================== softmax
    if constexpr (!PAGED) reg_inc<232>();
    const int r = tid;                                     // row of this CTA's half == TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const uint32_t s_tm = tmem + lane_base;
    const uint32_t o_tm = tmem + lane_base + Shape::kOCol;
    const int tl = (pk0 + rank * ROWS + r) / G;
    const int pos = sq.prefix + tl;
    const int vhi = p.is_cross ? sq.L - 1 : min(pos, sq.L - 1);
    const int vlo = p.window > 0 ? pos - p.window + 1 : 0;
    float m_ref = -INFINITY, l = 0.f;
    bool alive = true;
    const bool sc_neg = !(p.scale_log2 > 0.f);
    const float sc = sc_neg ? 1.f : p.scale_log2;

#pragma unroll 1
    for (int j = 0; j < ntiles; ++j) {
      const int sb = j & 1;
      alive = mbar_wait_warp_cluster(bar_s(sb), (j >> 1) & 1, abort_flag);
      if (!alive) break;
      tc_fence_after();
      const int k0 = kv_lo + j * BN;
      const bool need_mask = !(k0 >= vlo && k0 + BN - 1 <= vhi);
      uint32_t v[BN];
      tmem_ld32_at<0>(s_tm + sb * BN, v);
      tmem_ld32_at<32>(s_tm + sb * BN + 32, v);
      tmem_ld32_at<64>(s_tm + sb * BN + 64, v);
      tmem_ld32_at<96>(s_tm + sb * BN + 96, v);
      tmem_wait_ld();
      reg_fence(v);
      if (sc_neg) {  // a non-positive scale: fold it into the scores so that max() commutes
#pragma unroll
        for (int e = 0; e < BN; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * p.scale_log2);
      }
      if (need_mask) {
#pragma unroll
        for (int e = 0; e < BN; ++e) {
          const int kpos = k0 + e;
          if (!(kpos >= vlo && kpos <= vhi)) v[e] = 0xff800000u;  // -inf
        }
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int e = 0; e < BN; e += 8) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          mx[c] = max3(mx[c], __uint_as_float(v[e + 2 * c]), __uint_as_float(v[e + 2 * c + 1]));
      }
      const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc;
      // ---- lazy rescale of the accumulator
      float alpha = 1.f;
      bool resc = false;
      if (mt > m_ref + 8.f) {
        if (m_ref != -INFINITY) {
          alpha = fast_exp2(m_ref - mt);
          resc = true;
        }
        m_ref = mt;
      }
      if (j > 0 && __any_sync(0xffffffffu, resc)) {
        alive = mbar_wait_warp_cluster(bar_pv((j - 1) & 1), ((j - 1) >> 1) & 1, abort_flag);
        if (!alive) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(o_tm + c * 32, o);
          tmem_wait_ld();
          reg_fence(o);
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
          tmem_st32(o_tm + c * 32, o);
        }
        tmem_wait_st();
      }
      l *= alpha;
      const float nmu = (m_ref == -INFINITY) ? 0.f : -m_ref;
      // ---- P = exp2(s*scale - m_ref) as packed 16-bit pairs over the S columns
      const uint64_t sc2 = pack_f32x2(sc, sc), nmu2 = pack_f32x2(nmu, nmu);
      uint64_t la = pack_f32x2(0.f, 0.f), lb = la;
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t pk16[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float x0, x1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[c * 32 + e]), __uint_as_float(v[c * 32 + e + 1])),
                                 sc2, nmu2), x0, x1);
          const float p0 = fast_exp2(x0);
          const float p1 = fast_exp2(x1);
          if (e & 2) lb = add_f32x2(lb, pack_f32x2(p0, p1));
          else la = add_f32x2(la, pack_f32x2(p0, p1));
          pk16[e >> 1] = MmaOp<T>::pack(p0, p1);
        }
        tmem_st16(s_tm + sb * BN + c * 16, pk16);  // P columns [16c, 16c+16) of this S buffer
      }
      {
        float l0, l1;
        unpack_f32x2(add_f32x2(la, lb), l0, l1);
        l += l0 + l1;
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_at(bar_p(sb), 0);
    }

    // ---- epilogue: rows through the Q buffer (free: every S MMA is done), out as whole rows
    if (alive && ntiles > 0) {
      alive = mbar_wait_warp_cluster(bar_pv((ntiles - 1) & 1), ((ntiles - 1) >> 1) & 1, abort_flag);
      if (alive) tc_fence_after();
    }
    if (alive && warp * 32 < rows_valid) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      constexpr int RB = HD * 2;
      unsigned char* stage = smem_raw + (q_smem - smem_u32(smem_raw));
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t v[32];
        if (ntiles > 0) {
          tmem_ld32(o_tm + c * 32, v);
          tmem_wait_ld();
          reg_fence(v);
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = 0u;
        }
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          uint4 w;
          w.x = MmaOp<T>::pack(__uint_as_float(v[e]) * inv, __uint_as_float(v[e + 1]) * inv);
          w.y = MmaOp<T>::pack(__uint_as_float(v[e + 2]) * inv, __uint_as_float(v[e + 3]) * inv);
          w.z = MmaOp<T>::pack(__uint_as_float(v[e + 4]) * inv, __uint_as_float(v[e + 5]) * inv);
          w.w = MmaOp<T>::pack(__uint_as_float(v[e + 6]) * inv, __uint_as_float(v[e + 7]) * inv);
          const int chunk = c * 4 + (e >> 3);
          *reinterpret_cast<uint4*>(stage + r * RB + ((chunk ^ (r & 15)) << 4)) = w;
        }
      }
      __syncwarp();
      const int chunk = lane % CH;
#pragma unroll 8
      for (int rr = lane / CH; rr < 32; rr += 32 / CH) {
        const int row = warp * 32 + rr;
        if (row < rows_valid) {
          const int pkr = pk0 + rank * ROWS + row;
          const int tlr = pkr / G, gr = pkr - tlr * G;
          T* dst = static_cast<T*>(p.out) +
                   (static_cast<int64_t>(sq.q_begin + tlr) * p.hq + static_cast<int64_t>(h) * G + gr) * HD;
          uint4 w = *reinterpret_cast<const uint4*>(stage + row * RB + ((chunk ^ (row & 15)) << 4));
          if (p.gate) {
            const T* grow = static_cast<const T*>(p.gate) + (dst - static_cast<T*>(p.out));
            const uint4 gv = *reinterpret_cast<const uint4*>(grow + chunk * 8);
            T* wo = reinterpret_cast<T*>(&w);
            const T* wg = reinterpret_cast<const T*>(&gv);
#pragma unroll
            for (int e = 0; e < 8; ++e) wo[e] = apply_gate<T>(to_f32(wo[e]), wg[e]);
          }
          *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(dst) + chunk * 16) = w;
        }
      }
    }
    if (!alive && p.status && r == 0) atomicExch(p.status, 1);
  }

  // ---- teardown: both CTAs are past their last MMA, TMEM access and remote arrival
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();
  if (warp == Shape::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 512);
  }
}

}  // namespace msgl
