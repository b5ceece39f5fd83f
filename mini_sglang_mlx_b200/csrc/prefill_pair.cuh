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
// S has LA buffers and runs LA key tiles ahead of PV, so the softmax warps do not wait for the tensor
// pipe.  TMEM columns: S[b] at 128 b, O behind them: LA = 2 at head_dim 256, 3 at 128.
//
// At head_dim 128 two softmax groups take the tiles in turn: the 128 x 128 exponentials of a tile are
// 1024 cycles of the special-function unit, and one group alone needs 2140 for the tile (score load 240,
// row maximum 240, exponentials 1290, hand-over and waits 370), twice what the tensor pipe does.  Both
// add to one O, so a row's reference maximum goes from tile to tile: a group publishes it as soon as it
// has the tile's row maximum, and the other group, which is half a tile behind, picks it up.  (With an O
// and an S buffer for each group there is no third S buffer, and a group waits 1440 cycles per tile for
// PV and the next S: 1995 cycles per tile.)  At head_dim 256 one group keeps up with the tensor pipe (2048
// cycles per tile).
//
//   warps 0-3 (0-7)   softmax: thread r of a group owns row r of this CTA's half (TMEM lane r)
//   next warp         MMA issuer (leader)
//   next six warps    producers, three for the K tiles and three for the V tiles
//
// With per-token slots V comes by 16-byte copies, of four warps, and the warp that issues the MMAs in the
// leader hands the peer's over.  Everything else arrives by TMA and is counted in bytes on the leader's
// barrier, from both CTAs (.cta_group::2): full pages as boxes of 16 rows, anything else (per-token slots, a sequence's ragged
// last page, query rows whose heads do not divide 128) as tile::gather4 loads of four rows, where an
// absent row is one past the end of the tensor and reads as zeros.  Six producers because a warp
// issues one TMA instruction in about 67 cycles: with two, and the tiles announced to the leader by a
// relay warp, the MMA warp waited 1200 cycles per tile for K and V.
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
  static constexpr int kGroups = HD == 128 ? 2 : 1;       // softmax groups
  static constexpr int kMmaWarp = 4 * kGroups, kProducerWarp0 = kMmaWarp + 1;
  static constexpr int kKindWarps = 3;                    // producers of K, and of V
  static constexpr int kVWarps = PAGED ? 3 : 4;
  static constexpr int kWarps = kMmaWarp + 8;             // (whole warpgroups for setmaxnreg)
  // registers moved from the other warps to the softmax warps: 512 threads at 128, 384 at 168
  static constexpr int kSoftRegs = kGroups == 2 ? 192 : 200;
  static constexpr int kOtherRegs = kGroups == 2 ? 64 : 144;
  static constexpr int kThreads = kWarps * 32;
  static constexpr int kLA = kGroups == 2 ? 3 : 2;        // S buffers = tiles S runs ahead
  static constexpr int kOCol = kLA * kBN;
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
// Address of this shared-memory address in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t ra;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
  return ra;
}
// Arrivals on a barrier of either CTA, without memory ordering of their own (a release at cluster scope
// took 600 to 1300 cycles), for what is ordered otherwise: tensor memory by the tcgen05 fences on both
// sides, bytes that TMA counts by the barrier itself.  Ordinary writes to shared memory are neither:
// those of the peer are handed over by mbar_arrive_release_cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_release_cluster(uint32_t cluster_bar, uint32_t count) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_bar), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx_cluster(uint32_t cluster_bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_bar), "r"(bytes)
               : "memory");
}
// TMA into this CTA's shared memory, counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_pair_2d(uint32_t dst, const CUtensorMap* tmap, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(cluster_bar)
      : "memory");
}
__device__ __forceinline__ void tma_pair_3d(uint32_t dst, const CUtensorMap* tmap, int x, int y, int z,
                                            uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(z), "r"(cluster_bar)
      : "memory");
}
// four rows of 64 elements (one-row boxes), 512 bytes
__device__ __forceinline__ void tma_pair_gather4(uint32_t dst, const CUtensorMap* tmap, int x, const int (&rows)[4],
                                                 uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(rows[0]), "r"(rows[1]), "r"(rows[2]), "r"(rows[3]),
      "r"(cluster_bar)
      : "memory");
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

// A value and its tag as one 64-bit access: whoever sees the tag sees its value.  (The elements of a vector
// access of two words are accesses of their own, in no given order.)
__device__ __forceinline__ uint2 ld_shared_tagged(uint32_t addr) {
  uint64_t v;
  asm volatile("ld.volatile.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return make_uint2(static_cast<uint32_t>(v), static_cast<uint32_t>(v >> 32));
}
__device__ __forceinline__ void st_shared_tagged(uint32_t addr, uint32_t value, uint32_t tag) {
  asm volatile("st.volatile.shared.b64 [%0], %1;" ::"r"(addr), "l"(static_cast<uint64_t>(tag) << 32 | value)
               : "memory");
}
// Barrier of all threads of the CTA that may be reached from several places in the code.
template <int N>
__device__ __forceinline__ void cta_threads_sync() {
  asm volatile("bar.sync 2, %0;" ::"n"(N) : "memory");
}
// Barrier of the 256 threads of both softmax groups.
__device__ __forceinline__ void softmax_groups_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

struct PairBarriers {
  uint64_t q_full, full[8];              // leader: both CTAs' copies
  uint64_t empty[8];
  uint64_t v_here[4];                    // per-token slots: this CTA's half of a V tile (16-byte copies)
  uint64_t s_full[3], p_full[3], pv_done[3];
};

template <typename T, int HD, bool PAGED>
__global__ void __launch_bounds__(PairShape<HD, PAGED>::kThreads, 1)
    prefill_pair_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap tm_k,
                        const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tg_k,
                        const __grid_constant__ CUtensorMap tg_v, const __grid_constant__ CUtensorMap tm_q) {
  using Shape = PairShape<HD, PAGED>;
  constexpr int BM = Shape::kBM, BN = Shape::kBN, ROWS = Shape::kRows, NB = Shape::kBufs;
  constexpr int KEYS = BN / 2;                  // keys of a K tile in this CTA
  constexpr int CH = HD / 8;                    // 16-byte chunks of a token row
  constexpr int NKW = Shape::kKindWarps;
  constexpr int NG = Shape::kGroups, LA = Shape::kLA;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ PairBarriers bars;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ FoundItem found;
  __shared__ float2 s_ml[NG == 2 ? 2 * ROWS : 1];        // (reference maximum, sum) of the rows, per group
  // reference maxima after the even / odd tiles, each with its tile's number
  __shared__ __align__(16) uint2 s_mref[NG == 2 ? 2 * ROWS : 1];

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int G = p.group;
  const int rank = static_cast<int>(cluster_rank());

  auto bar_full = [&](int bf) { return smem_u32(&bars.full[bf]); };
  auto bar_empty = [&](int bf) { return smem_u32(&bars.empty[bf]); };
  auto bar_s = [&](int b) { return smem_u32(&bars.s_full[b]); };
  auto bar_p = [&](int b) { return smem_u32(&bars.p_full[b]); };
  auto bar_pv = [&](int b) { return smem_u32(&bars.pv_done[b]); };
  const uint32_t bar_q = smem_u32(&bars.q_full);
  // (every second buffer of the ring holds V tiles, so a barrier's next use is behind the buffer's)
  auto bar_v = [&](int tile) { return smem_u32(&bars.v_here[tile % (NB / 2)]); };

  // ---- set-up, a warp for each part of it
  if (warp == Shape::kMmaWarp) {
    tmem_alloc_pair(smem_u32(&s_tmem_base), 512);
    tmem_relinquish_pair();
  }
  if (warp == 1) {
    // a barrier per lane
    auto init = [&](uint64_t* first, int n, int count) {
      if (lane < n) mbar_init(smem_u32(first + lane), count);
    };
    init(&bars.q_full, 1, 2 * 2 * NKW);
    init(bars.full, NB, 2 * NKW);            // both CTAs' producers (V of per-token slots: the peer's relay)
    init(bars.empty, NB, 1);
    if (!PAGED) init(bars.v_here, NB / 2, Shape::kVWarps * 32);
    init(bars.s_full, LA, 1);
    init(bars.p_full, LA, 2 * (ROWS / 32));
    init(bars.pv_done, LA, 1);
    if (lane == 0) s_abort = 0;
    fence_mbar_init();
  }
  if (NG == 2 && tid < 2 * ROWS) s_mref[tid] = make_uint2(0u, 0xffffffffu);
  if (!p.early) grid_dependency_wait();
  if (p.batch <= kWarpBatchMax) {
    if (warp == 0) find_item_warp(p, static_cast<int>(blockIdx.x) / 2, BM, &found);
  } else {
    ItemCoord at;
    const bool have = find_item<Shape::kThreads>(p, static_cast<int>(blockIdx.x) / 2, BM,
                                                 reinterpret_cast<int*>(smem_raw), at);
    fence_proxy_async_smem();   // (Q comes to where the item search had its counts)
    if (tid == 0) {
      found.have = have;
      if (have) {
        found.at = at;
        found.seq = load_seq_shape(p, at.b, BM);
      }
    }
  }
  tc_fence_before();
  cluster_sync_all();           // the barriers of both CTAs exist (and the CTA's own set-up is done)
  tc_fence_after();
  const uint32_t tmem = s_tmem_base;
  const bool producer = warp >= Shape::kProducerWarp0 && warp < Shape::kProducerWarp0 + NKW + Shape::kVWarps;
  if (p.early && !(producer && found.have)) grid_dependency_wait();   // (producers: once they know their first copies)
  if (!p.early || warp == 0) grid_dependency_launch();
  if (!found.have) {            // the same in both CTAs: a launch rank past the last item
    if (warp == Shape::kMmaWarp) tmem_dealloc_pair(tmem, 512);
    return;
  }
  const ItemCoord it = found.at;
  const int h = it.h;
  const SeqShape sq = found.seq;
  auto over_group = [&](int x) { return divide_by(x, p.group_recip); };
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
  const int tok_first = over_group(pk0);
  const int tok_last = over_group(pk0 + rows_pair - 1);
  int kv_lo = p.window > 0 ? max(0, sq.prefix + tok_first - p.window + 1) : 0;
  kv_lo = (kv_lo / BN) * BN;
  const int kv_hi = p.is_cross ? sq.L : min(sq.L, sq.prefix + tok_last + 1);   // keys from here on are never read
  const int ntiles = kv_hi > kv_lo ? ceil_div(kv_hi - kv_lo, BN) : 0;

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem0;
  const uint32_t ring = smem0 + Shape::kQBytes;
  volatile int* abort_flag = &s_abort;

  // Output rows are packed in the Q buffer (free then: every S MMA is done; chunk c of row r sits at chunk
  // position c ^ (r & 15)) and leave as whole rows, by all warps of the CTA, each with four of the gate's reads
  // in flight from before the last PV is done.  (Of 53000 cycles of a gated pair at head_dim 256, 12400 went here with
  // two reads at a time and one element per instruction.)
  constexpr int RB = HD * 2;
  unsigned char* stage = smem_raw + (q_smem - smem_u32(smem_raw));
  constexpr int RPI = 32 / CH;                                // rows of a warp's access
  constexpr int STEP = Shape::kWarps * RPI, FLY = 4;          // the gate's reads run FLY accesses ahead
  uint4 gv[FLY];
  auto row_offset = [&](int row) -> int64_t {
    const int pk = pk0 + rank * ROWS + row;
    const int tl = over_group(pk), g = pk - tl * G;
    return (static_cast<int64_t>(sq.q_begin + tl) * p.hq + static_cast<int64_t>(h) * G + g) * HD + lane % CH * 8;
  };
  auto read_gate = [&](int row, uint4& g) {
    if (p.gate && row < rows_valid) g = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.gate) + row_offset(row));
  };
  auto first_gates = [&]() {
#pragma unroll
    for (int f = 0; f < FLY; ++f) read_gate(warp * RPI + lane / CH + f * STEP, gv[f]);
  };
  auto write_rows = [&]() {
    cta_threads_sync<Shape::kThreads>();
    if (s_abort != 0) return;
    const int chunk = lane % CH;
#pragma unroll 1
    for (int r0 = warp * RPI + lane / CH; r0 < rows_valid; r0 += FLY * STEP) {
#pragma unroll
      for (int f = 0; f < FLY; ++f) {
        const int row = r0 + f * STEP;
        if (row >= rows_valid) break;
        uint4 w = *reinterpret_cast<const uint4*>(stage + row * RB + ((chunk ^ (row & 15)) << 4));
        if (p.gate) {
          w.x = apply_gate_pair<T>(w.x, gv[f].x);
          w.y = apply_gate_pair<T>(w.y, gv[f].y);
          w.z = apply_gate_pair<T>(w.z, gv[f].z);
          w.w = apply_gate_pair<T>(w.w, gv[f].w);
          read_gate(row + FLY * STEP, gv[f]);
        }
        *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + row_offset(row)) = w;
      }
    }
  };

  if (warp >= Shape::kMmaWarp) {
    reg_dec<Shape::kOtherRegs>();
    if (warp >= Shape::kProducerWarp0 && warp < Shape::kProducerWarp0 + NKW + Shape::kVWarps) {
      // =========================================================== producers
      const int pid = warp - Shape::kProducerWarp0;
      const bool is_k = pid < NKW;
      const int pw = is_k ? pid : pid - NKW;            // among the warps of its kind
      const uint32_t q_bar = cluster_addr(bar_q, 0);
      if (lane == 0) {
        prefetch_tensormap(&tm_q);
        prefetch_tensormap(is_k ? &tg_k : &tg_v);
        if (PAGED) prefetch_tensormap(is_k ? &tm_k : &tm_v);
      }
      bool waited = !p.early;
      auto wait_in_front = [&]() {
        if (waited) return;
        waited = true;
        grid_dependency_wait();
      };
      // ---- Q, dealt to all producers: boxes of 64 columns x 128 rows where a box holds whole tokens
      // (rows past the sequence's last query token hold a neighbour's rows then: computed on, never
      // written), else four rows at a time
      auto load_q = [&]() {
        if (pid >= 2 * NKW) return;
        if (p.q_tma) {
          if (elect_one()) {
            int mine = 0;
            for (int c = pid; c < HD / 64; c += 2 * NKW) ++mine;
            mbar_arrive_expect_tx_cluster(q_bar, mine * (ROWS * 128));
            for (int c = pid; c < HD / 64; c += 2 * NKW)
              tma_pair_3d(q_smem + c * (ROWS * 128), &tm_q, c * 64, h * G, sq.q_begin + tok_first + rank * (ROWS / G), q_bar);
          }
        } else {
          // lane l knows the rows 4 l .. 4 l + 3; the groups l = pid, pid + 6, ... are this warp's
          int rows[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = lane * 4 + e;
            const int pk = pk0 + rank * ROWS + row;
            const int tl = over_group(pk), g = pk - tl * G;
            rows[e] = row < rows_valid ? (sq.q_begin + tl) * p.hq + h * G + g : p.total_q * p.hq;
          }
          if (elect_one()) mbar_arrive_expect_tx_cluster(q_bar, (32 - pid + 2 * NKW - 1) / (2 * NKW) * (HD * 8));
          __syncwarp();
#pragma unroll 1
          for (int l = pid; l < 32; l += 2 * NKW) {
            int r4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) r4[e] = __shfl_sync(0xffffffffu, rows[e], l);
            if (elect_one()) {
#pragma unroll
              for (int c = 0; c < HD / 64; ++c)
                tma_pair_gather4(q_smem + c * (ROWS * 128) + l * 512, &tm_q, c * 64, r4, q_bar);
            }
            __syncwarp();
          }
        }
        __syncwarp();
      };
      // ---- key tiles.  K: this CTA's 64 keys, all columns; V: all 128 keys, its half of the columns.
      const int absent = static_cast<int>(p.num_slots);
      const int32_t* ids = (PAGED ? p.page_indices : p.kv_indices) + sq.kv_begin;
      const uint32_t full0 = cluster_addr(bar_full(0), 0);
      bool alive = true;
      auto produce = [&](auto kind, const CUtensorMap* tm, const CUtensorMap* tg) {
        constexpr bool K = decltype(kind)::value;
        constexpr int RT = K ? KEYS : BN;                         // rows of the tile copied here
        constexpr int COLS = K ? HD / 64 : HD / 128;              // blocks of 64 columns
        // what is dealt to the warps: boxes, or groups of four rows with all their column blocks
        constexpr int UNITS = PAGED ? RT / kTmaBoxRows * COLS : RT / 4;
        constexpr int MINE = (UNITS + NKW - 1) / NKW;             // of this warp: pw, pw + NKW, ...
        constexpr int UB = PAGED ? kTmaBoxRows * 128 : 512 * COLS;     // bytes
        const uint32_t my_bytes = static_cast<uint32_t>((UNITS - pw + NKW - 1) / NKW) * UB;
        const int x0 = h * HD + (K ? 0 : rank * (HD / 2));
        const int key0 = K ? rank * KEYS : 0;                     // first key of the tile copied here
        // PAGED: lane i = page i of the copied keys: a = its first pool row, n = rows of it that belong
        // to the sequence.  Per-token: lane l = keys 4 l .. 4 l + 3: their slots.
        struct Ids {
          int a[PAGED ? 1 : 4], n;
        };
        auto fetch = [&](int tile, Ids& d) {
          const int t0 = kv_lo + tile * BN + key0;
          if constexpr (PAGED) {
            d.a[0] = absent;
            d.n = 0;
            const int t = t0 + lane * kTmaBoxRows;
            if (lane * kTmaBoxRows < RT && tile < ntiles && t < kv_hi) {
              const int page = divide_by(t, p.page_recip);
              const int pg = __ldg(ids + page);
              const int64_t row0 = static_cast<int64_t>(pg) * p.page_size + (t - page * p.page_size);
              const int nv = min(kTmaBoxRows, sq.L - t);
              if (pg < 0 || row0 + nv > p.num_slots) {
                if (p.status) atomicExch(p.status, 2);     // page outside the pool: rows read as zeros
              } else {
                d.a[0] = static_cast<int>(row0);
                d.n = nv;
              }
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int t = t0 + lane * 4 + e;
              int slot = -1;
              if (lane * 4 < RT && tile < ntiles && t < kv_hi) {
                slot = __ldg(ids + t);
                if ((slot < -1 || static_cast<int64_t>(slot) >= p.num_slots) && p.status) atomicExch(p.status, 2);
              }
              d.a[e] = slot < 0 || static_cast<int64_t>(slot) >= p.num_slots ? absent : slot;
            }
          }
        };
        Ids cur, nxt;
        fetch(0, cur);
        wait_in_front();
        if (!K && ntiles > 0) load_q();
#pragma unroll 1
        for (int t = 0; t < ntiles; ++t) {
          fetch(t + 1, nxt);                                      // in flight while this tile's copies are issued
          const int seq = K ? ring_seq_k<LA>(t) : ring_seq_v<LA>(t);
          const int bf = seq % NB;
          alive = mbar_wait_warp(bar_empty(bf), ((seq / NB) & 1) ^ 1, abort_flag);
          if (!alive) break;
          const uint32_t dst = ring + bf * Shape::kBufBytes;
          const uint32_t bar = full0 + bf * 8;
          if (elect_one()) mbar_arrive_expect_tx_cluster(bar, my_bytes);
          __syncwarp();
#pragma unroll(PAGED ? MINE : 2)
          for (int k = 0; k < MINE; ++k) {
            const int id = pw + k * NKW;
            if (UNITS % NKW != 0 && id >= UNITS) break;
            if constexpr (PAGED) {
              constexpr int PAGES = RT / kTmaBoxRows;
              const int i = id % PAGES, c = id / PAGES;
              const uint32_t at = dst + c * (RT * 128) + i * UB;
              const int y = __shfl_sync(0xffffffffu, cur.a[0], i), n = __shfl_sync(0xffffffffu, cur.n, i);
              if (elect_one()) {
                if (n == kTmaBoxRows) {
                  tma_pair_2d(at, tm, x0 + c * 64, y, bar);
                } else {
#pragma unroll 1
                  for (int r = 0; r < kTmaBoxRows; r += 4) {
                    int r4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) r4[e] = r + e < n ? y + r + e : absent;
                    tma_pair_gather4(at + r * 128, tg, x0 + c * 64, r4, bar);
                  }
                }
              }
            } else {
              int r4[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) r4[e] = __shfl_sync(0xffffffffu, cur.a[e], id);
              if (elect_one()) {
#pragma unroll
                for (int c = 0; c < COLS; ++c) tma_pair_gather4(dst + c * (RT * 128) + id * 512, tg, x0 + c * 64, r4, bar);
              }
            }
            __syncwarp();
          }
          cur = nxt;
          if (K && t == 0) load_q();      // (behind the first tile, whose page ids were on their way longer)
        }
      };
      if (is_k) {
        produce(std::true_type{}, &tm_k, &tg_k);
      } else if constexpr (PAGED) {
        produce(std::false_type{}, &tm_v, &tg_v);
      } else {
        // V of per-token slots: 16-byte copies, the other path into shared memory (a gather of four
        // 128-byte rows takes about 66 cycles of TMA, a copy instruction of 512 bytes about 47 of the
        // load/store unit: K by one and V by the other nearly add up).  They are ordinary writes: a tile's
        // copies arrive on a barrier of this CTA as they land, and who hands them to the tensor pipe
        // (the leader its own half, the relay below the peer's) puts the proxy fence behind it.
        constexpr int VCH = CH / 2;                               // 16-byte chunks of half a row
        constexpr int RPA = 32 / VCH;                             // rows of an access
        const unsigned char* vbase = static_cast<const unsigned char*>(p.v_cache) + static_cast<int64_t>(h) * (HD * 2) + rank * HD;
        const int64_t slot_stride = static_cast<int64_t>(p.hkv) * (HD * 2);
        const int row0 = pw * 32;                                 // 32 of the tile's 128 keys
        auto slot_of = [&](int tile) -> int {
          const int t = kv_lo + tile * BN + row0 + lane;
          int slot = tile < ntiles && t < kv_hi ? __ldg(ids + t) : -1;
          if (slot < -1 || static_cast<int64_t>(slot) >= p.num_slots) {
            if (p.status) atomicExch(p.status, 2);
            slot = -1;
          }
          return slot;
        };
        int slot = slot_of(0);
        wait_in_front();
        if (ntiles > 0) load_q();
#pragma unroll 1
        for (int t = 0; t < ntiles; ++t) {
          const int next = slot_of(t + 1);
          const int seq = ring_seq_v<LA>(t), bf = seq % NB;
          alive = mbar_wait_warp(bar_empty(bf), ((seq / NB) & 1) ^ 1, abort_flag);
          if (!alive) break;
          const uint32_t dst = ring + bf * Shape::kBufBytes;
          const int chunk = lane % VCH;
#pragma unroll
          for (int i = 0; i < 32 / RPA; ++i) {
            const int row = i * RPA + lane / VCH;
            const int sl = __shfl_sync(0xffffffffu, slot, row);
            cp_async_16(dst + tc_tile_offset<BN>(row0 + row, chunk),
                        vbase + (sl >= 0 ? sl * slot_stride : 0) + chunk * 16, sl >= 0 ? 16 : 0);
          }
          cp_async_mbar_arrive(bar_v(t));
          slot = next;
        }
        cp_async_wait_all();
      }
      if (!alive) {
        if (p.status && lane == 0) atomicExch(p.status, 1);
        // gave up: let the copies still in flight land before the shared memory goes away
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
      }
    } else if (warp == Shape::kMmaWarp && rank == 0) {
      // =========================================================== MMA issuer
      const uint32_t idesc_s = idesc_m256<T>(BN, 0);
      const uint32_t idesc_pv = idesc_m256<T>(HD, 1);
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t desc_k = smem_desc_sw128(0, 16, 1024);                 // Q / K: K-major
      const uint64_t desc_v = smem_desc_sw128(0, BN * 128, 1024);           // V: MN-major
      const int last_seq = ring_seq_v<LA>(ntiles - 1);
      bool alive = true;
      auto acquire = [&](int seq) {
        alive = mbar_wait_warp(bar_full(seq % NB), (seq / NB) & 1, abort_flag);
        if (alive) tc_fence_after();
      };
      // V of per-token slots: the copies of this CTA's threads, and those of the peer's by its relay
      auto acquire_written = [&](int seq, int tile) {
        alive = mbar_wait_warp(bar_v(tile), (tile / (NB / 2)) & 1, abort_flag) &&
                mbar_wait_warp<true>(bar_full(seq % NB), (seq / NB) & 1, abort_flag);
        if (alive) {
          fence_proxy_async_smem();
          tc_fence_after();
        }
      };
      // frees a ring buffer in both CTAs (only while somebody will fill it again)
      auto release = [&](int seq) {
        if (seq + NB <= last_seq) tc_commit_pair(bar_empty(seq % NB));
      };
      if (ntiles > 0) alive = mbar_wait_warp(bar_q, 0, abort_flag);
#pragma unroll 1
      for (int j = -LA; j < ntiles && alive; ++j) {
        const bool do_pv = j >= 0, do_s = j + LA < ntiles;
        const int sv = ring_seq_v<LA>(j), sk = ring_seq_k<LA>(j + LA);
        const int sb = (j + LA) % LA;                       // buffer of P of tile j and of S of tile j + LA
        if (do_pv) {
          if constexpr (PAGED) acquire(sv);
          else acquire_written(sv, j);
        }
        if (alive && do_s) acquire(sk);
        if (alive && do_pv) {
          alive = mbar_wait_warp(bar_p(sb), (j / LA) & 1, abort_flag);
          tc_fence_after();
        }
        if (!alive) break;
        const uint32_t vb = (ring + (do_pv ? sv % NB : 0) * Shape::kBufBytes) >> 4;
        const uint32_t kb = (ring + (do_s ? sk % NB : 0) * Shape::kBufBytes) >> 4;
        const uint32_t qa = q_smem >> 4;
        const uint32_t o_tm = tmem_u + Shape::kOCol;
        const uint32_t ps_tm = tmem_u + sb * BN;
        if (elect_one()) {
          if (do_pv) {
#pragma unroll
            for (int ks = 0; ks < BN / 16; ++ks)
              tc_mma_pair_ts(o_tm, ps_tm + ks * 8, desc_v | (vb + ks * (2048 >> 4)), idesc_pv,
                             (j == 0 && ks == 0) ? 0u : 1u);
            tc_commit_pair(bar_pv(sb));
            release(sv);
          }
          if (do_s) {
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
              const uint32_t qoff = ((ks >> 2) * (ROWS * 128) + (ks & 3) * 32) >> 4;
              const uint32_t koff = ((ks >> 2) * (KEYS * 128) + (ks & 3) * 32) >> 4;
              tc_mma_pair_ss(ps_tm, desc_k | (qa + qoff), desc_k | (kb + koff), idesc_s, ks > 0 ? 1u : 0u);
            }
            tc_commit_pair(bar_s(sb));
            release(sk);
          }
        }
        __syncwarp();
      }
      if (!alive && p.status && lane == 0) atomicExch(p.status, 1);
    } else if (!PAGED && warp == Shape::kMmaWarp) {
      // =========================================================== relay of the peer's V copies
      // The release at cluster scope that ordinary writes need in front of the leader's MMAs.  A warp without
      // copies of its own gives it: a release waits for its thread's copies in flight (given by the copying
      // warps, behind the next tile's copies, it took 414 us instead of 280 on 1024 tokens over 16000 at
      // head_dim 256, 455 instead of 394 on the gated prompts).
      const uint32_t full0 = cluster_addr(bar_full(0), 0);
      bool alive = true;
#pragma unroll 1
      for (int t = 0; t < ntiles && alive; ++t) {
        alive = mbar_wait_warp(bar_v(t), (t / (NB / 2)) & 1, abort_flag);
        fence_proxy_async_smem();
        if (alive && lane == 0) mbar_arrive_release_cluster(full0 + ring_seq_v<LA>(t) % NB * 8, 2 * NKW);
      }
      if (!alive && p.status && lane == 0) atomicExch(p.status, 1);
    }
    __syncwarp();
    first_gates();
    write_rows();
  } else {
    // =========================================================== softmax
    reg_inc<Shape::kSoftRegs>();
    const int grp = warp >> 2;                             // takes tiles grp, grp + NG, ...
    const int r = tid & (ROWS - 1);                        // row of this CTA's half == TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_tm = tmem + lane_base;
    const uint32_t o_tm = tmem + lane_base + Shape::kOCol;
    const int tl = over_group(pk0 + rank * ROWS + r);
    const int pos = sq.prefix + tl;
    const int vhi = p.is_cross ? sq.L - 1 : min(pos, sq.L - 1);
    const int vlo = p.window > 0 ? pos - p.window + 1 : 0;
    float m_ref = -INFINITY, l = 0.f;
    bool alive = true;
    const bool sc_neg = !(p.scale_log2 > 0.f);
    const float sc = sc_neg ? 1.f : p.scale_log2;

    const uint32_t p_bar = cluster_addr(bar_p(0), 0);
    // the gate's rows on their way into L2: the epilogue wants them
    if (p.gate) {
      for (int e = warp * 32 + lane; e < rows_valid * (HD / 64); e += NG * ROWS) {
        const int pk = pk0 + rank * ROWS + e / (HD / 64);
        const int tle = over_group(pk), g = pk - tle * G;
        prefetch_l2(static_cast<const T*>(p.gate) +
                    (static_cast<int64_t>(sq.q_begin + tle) * p.hq + static_cast<int64_t>(h) * G + g) * HD +
                    e % (HD / 64) * 64);
      }
    }
#pragma unroll 1
    for (int j = grp; j < ntiles; j += NG) {
      const int sb = j % LA;
      alive = mbar_wait_warp(bar_s(sb), (j / LA) & 1, abort_flag);
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
        if constexpr (HD == 128) {
          // visible keys as bits, 32 at a time: predicates from a register, not two comparisons per key (six short
          // prompts, 8 layers: 106.7 us for 112.1; at head_dim 256 it is the other way round, 159 for 147)
          const int hi = vhi - k0, lo = vlo - k0;             // lo <= e <= hi
#pragma unroll
          for (int c = 0; c < BN / 32; ++c) {
            const int h32 = hi - 32 * c, l32 = lo - 32 * c;
            const uint32_t below = h32 >= 31 ? ~0u : h32 < 0 ? 0u : (2u << h32) - 1u;
            const uint32_t from = l32 <= 0 ? ~0u : l32 > 31 ? 0u : ~0u << l32;
            const uint32_t seen = below & from;
#pragma unroll
            for (int e = 0; e < 32; ++e) v[32 * c + e] = seen >> e & 1u ? v[32 * c + e] : 0xff800000u;  // -inf
          }
        } else {
#pragma unroll
          for (int e = 0; e < BN; ++e) {
            const int kpos = k0 + e;
            if (!(kpos >= vlo && kpos <= vhi)) v[e] = 0xff800000u;  // -inf
          }
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
      // ---- the row's reference maximum: the one after tile j - 1, raised (and O rescaled) only when the
      // maximum has grown by more than 2^8
      float alpha = 1.f;                      // of this group's sum
      float m_old = m_ref;
      if constexpr (NG == 2) {
        if (j > 0) {
          // (a value tagged with its tile: the reader polls its own row, no barrier in between)
          const uint32_t at = smem_u32(&s_mref[((j - 1) & 1) * ROWS + r]);
          uint2 got = ld_shared_tagged(at);
          if (got.y != static_cast<uint32_t>(j - 1)) {
            const long long t0 = clock64();
            while ((got = ld_shared_tagged(at)).y != static_cast<uint32_t>(j - 1)) {
              if (*abort_flag != 0 || clock64() - t0 > kTcWaitCycles) {
                *abort_flag = 1;
                alive = false;
                break;
              }
            }
          }
          alive = __all_sync(0xffffffffu, alive ? 1 : 0) != 0;
          if (!alive) break;
          m_old = __uint_as_float(got.x);
        }
      }
      const float m_new = mt > m_old + 8.f ? mt : m_old;
      if constexpr (NG == 2) {
        st_shared_tagged(smem_u32(&s_mref[(j & 1) * ROWS + r]), __float_as_uint(m_new), j);
      }
      if (m_new != m_ref && m_ref != -INFINITY) alpha = fast_exp2(m_ref - m_new);
      const bool resc = m_new != m_old && m_old != -INFINITY;
      const float o_scale = resc ? fast_exp2(m_old - m_new) : 1.f;
      m_ref = m_new;
      if (j > 0 && __any_sync(0xffffffffu, resc)) {
        alive = mbar_wait_warp(bar_pv((j - 1) % LA), ((j - 1) / LA) & 1, abort_flag);
        if (!alive) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(o_tm + c * 32, o);
          tmem_wait_ld();
          reg_fence(o);
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * o_scale);
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
          const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(v[c * 32 + e]), __uint_as_float(v[c * 32 + e + 1])), sc2, nmu2);
          float x0, x1;
          unpack_f32x2(x, x0, x1);
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
      if (lane == 0) mbar_arrive_cluster(p_bar + sb * 8);
    }

    // ---- epilogue
    const bool any = ntiles > 0;
    first_gates();
    if (alive && any) {
      alive = mbar_wait_warp(bar_pv((ntiles - 1) % LA), ((ntiles - 1) / LA) & 1, abort_flag);
      if (alive) tc_fence_after();
    }
    float inv = l > 0.f ? 1.f / l : 0.f;
    if constexpr (NG == 2) {
      // O is relative to the last tile's reference maximum, each group's sum to that of its own last tile
      s_ml[grp * ROWS + r] = make_float2(m_ref, l);
      softmax_groups_sync();
      const float2 peer = s_ml[(grp ^ 1) * ROWS + r];
      const float M = fmaxf(m_ref, peer.x);   // (it only grows)
      const float L = (m_ref == -INFINITY ? 0.f : l * fast_exp2(m_ref - M)) +
                      (peer.x == -INFINITY ? 0.f : peer.y * fast_exp2(peer.x - M));
      inv = L > 0.f ? 1.f / L : 0.f;
    }
#pragma unroll 1
    for (int c = grp * (HD / 32 / NG); c < (grp + 1) * (HD / 32 / NG); ++c) {   // a group's share of the columns
      uint32_t v[32];
      if (any && alive) {
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
    write_rows();
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
