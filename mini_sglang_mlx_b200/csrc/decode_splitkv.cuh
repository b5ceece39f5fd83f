// Split-KV flash-decoding for one query token per sequence (sm_100a).
//
// Work split.  For every KV head the sequences' 16-token groups are laid end to end and cut into equal
// shares; a CTA owns one share of one head and walks it across sequence boundaries (each warp finds the
// share's first sequence with a warp scan of the lengths).  Shares give every CTA the same
// amount of K/V however ragged the batch is: with one CTA per (sequence, head, split) a batch of 37
// sequences of 100 .. 6000 tokens needed 4.8 waves of CTAs, each a chain of latencies (60 us against
// 23 us of K/V traffic).  CTAs of neighbouring heads run together, so that a page's rows of all
// heads, which are adjacent in the pool, are fetched at about the same time.
//
// Inside a CTA the G = Hq/Hkv query heads of the KV head are the rows of a 16-row tensor-core tile;
// the share's 16-token groups go round-robin to the warps, each through a warp-private ring of
// swizzled shared-memory tiles that runs on across sequence boundaries.  S = Q K^T and O += P V run
// as m16n8k16 mma.sync with fp32 accumulation and a base-2 online softmax whose row reductions are
// warp shuffles.  (mma.sync, not tcgen05: the operator is bound by HBM, and a 16-row tile would
// leave 7/8 of a 128-row tile idle.)
//
// A part of a sequence that a share holds is a segment.  At its end the warps' (max, sum, O) are
// merged through shared memory, a warp per query head; a segment that is a whole sequence writes the final
// rows, any other (the first and the last of a share at most) writes an fp32 partial (sum of the weighted rows,
// maximum, sum of the weights) to scratch.  A warp of a CTA that is through with its share arrives at the
// counters of the heads whose partials it wrote, and the one that arrives last at a head merges its pieces;
// there is no second launch and no barrier.
//
// What bounds a small call is none of the chip's rates but the chain of a CTA's instructions, each of which
// waits for the one in front (one warp per scheduler: 8 to 10 cycles per instruction, 2320 of them on 700 tokens of one
// sequence, 2975 before; memory 10 % of it).  So the search for the share has no divisions and one scan, new rows' slots are
// held in registers, and the merge of the pieces reads them straight into registers.
//
// Per-token form: K and V rows (256 or 512 bytes per token and head) are gathered through the slot
// ids with 16-byte cp.async copies.  Page-granular form (PAGED): a group is one page (or a 16-row
// slice of a larger page), contiguous in the pool, so lane 0 fetches it with a TMA box copy each for K and V
// (cp.async.bulk.tensor.3d: HD / 64 blocks of 16 rows x 64 elements, 128-byte swizzle) straight from the page id and
// the warp waits on the stage's mbarrier; only a sequence's ragged last page is copied row by row
// (rows past the length are zero-filled).
//
// Semantics follow the reference stages
// (mini-sglang-mlx-kernel/csrc/paged_decode_attention.metal:313-506 and
// 512-586): slot addressing row = kv_indices[kv_indptr[b] + t]; its partials are normalised, each with a
// log-sum-exp, here they carry (maximum in log2 units, sum) and are divided once, in the merge:
// out = sum_s 2^{M_s-M} O_s / sum_s 2^{M_s-M} l_s.  The reference's split counts are hints; here the shares take their place
// (its result does not depend on them).  Address arithmetic is 64-bit.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace msgl {

struct DecodeParams {
  const void* q;
  const void* k_cache;
  const void* v_cache;
  // per-token form: kv_indptr / kv_indices; page-granular (kv_lens != null): page_indptr / page_indices
  const int32_t* indptr;
  const int32_t* indices;
  const int32_t* kv_lens;
  int page_size;
  void* out;
  const void* gate;  // (batch, hq, D) or null: out *= sigmoid(gate)
  float* part;       // (slots, group, decode_partial_floats(D)): partials, each with (maximum, sum) behind it
  // (batch, hq) arrival counters of a (sequence, query head)'s segments: the warp that arrives last
  // merges the partials and puts the counter back to zero.  Zero before the first launch.
  int* tickets;
  int* status;       // device status word (0 = ok); may be null
  int batch, hq, hkv, group;
  int num_shares;    // shares per head at most (= gridDim.x / hkv); 0: a share is a whole sequence
  int wave;          // shares per head that fill the GPU once
  float inv_wave;    // 1 / wave, not below it
  int max_waves;     // num_shares / wave
  int min_share, max_share;  // groups a share holds at least; at most, while num_shares allows another wave
  int pad;           // what the end of a segment costs, in groups
  int max_pieces;    // pieces of a sequence up to which the shares do not grow with the merge
  float merge_row;   // what merging a piece costs, in groups
  int64_t num_slots;
  float scale_log2;  // sm_scale * log2(e)
  // The call's own K/V store is the kernel in front in the stream: it writes the pool rows
  // new_slots[0 .. num_new) (and q, if it rotates it), and everything before it is complete when
  // this kernel starts.  num_new < 0: nothing is known about the kernel in front.
  const int32_t* new_slots;
  int num_new;
};
constexpr int kDecodeNewMax = 128;      // new rows at most that a warp compares its first groups with

constexpr int kDecodeGroupTokens = 16;  // tokens a warp consumes per step

// Shared memory of a CTA: ring, alignment slack of the TMA tiles, merge rows, (m, l) of the merge, two
// windows of sequences per warp, at head_dim 256 the query rows.
constexpr int kDecodeMergeHeads = 4;    // query heads merged at a time
__host__ __device__ constexpr int decode_merge_row_floats(int hd) { return hd + 8; }  // (+8: bank-conflict-free)
__host__ __device__ constexpr int decode_partial_floats(int hd) { return hd + 4; }    // (rows of 16-byte multiples)
__host__ __device__ constexpr int decode_smem_bytes(int hd, int warps, int stages) {
  return warps * stages * 2 * kDecodeGroupTokens * hd * 2 + 1024 +
         warps * kDecodeMergeHeads * decode_merge_row_floats(hd) * 4 + warps * 16 * 2 * 4 + warps * 64 * 16 +
         (hd == 256 ? 16 * hd * 2 : 0);
}

// A lane's VPL gate values of an output row (a call without a gate has none), read as one vector.
template <typename T, int VPL>
struct GateVec {
  typename std::conditional<VPL == 4, uint2, uint4>::type bits;
  bool on;
  __device__ __forceinline__ void load(const T* gate, int64_t at) {
    on = gate != nullptr;
    if (on) bits = *reinterpret_cast<const decltype(bits)*>(gate + at);
  }
};

// VPL consecutive output columns of a lane, gated if the call has a gate.
template <typename T, int VPL>
__device__ __forceinline__ void write_decode_row(T* out, const GateVec<T, VPL>& gate, int64_t at,
                                                 const float (&x)[VPL]) {
  alignas(16) T vals[VPL];
  const T* gv = reinterpret_cast<const T*>(&gate.bits);
#pragma unroll
  for (int e = 0; e < VPL; ++e) vals[e] = gate.on ? apply_gate<T>(x[e], gv[e]) : MmaOp<T>::from_float(x[e]);
  *reinterpret_cast<decltype(gate.bits)*>(out + at) = *reinterpret_cast<const decltype(gate.bits)*>(vals);
}

template <typename T, int HD, int NWARPS, int NSTAGES, bool PAGED>
__global__ void __launch_bounds__(NWARPS * 32, HD == 256 ? 1 : 2)
    decode_kernel(const DecodeParams p, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v) {
  constexpr int CH = HD / 8;                              // 16-byte chunks per token row
  constexpr int ROW_BYTES = HD * 2;
  constexpr int TILE_BYTES = kDecodeGroupTokens * ROW_BYTES;  // one K (or V) group tile
  constexpr int KSTEPS = HD / 16;
  constexpr int NT = HD / 8;                              // output n-tiles
  constexpr int MROW = decode_merge_row_floats(HD);
  constexpr int PROW = decode_partial_floats(HD);
  static_assert(CH == 16 || CH == 32, "head_dim must be 128 or 256");
  static_assert(NWARPS == kDecodeMergeHeads, "a warp merges a head");

  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t s_bar[PAGED ? NWARPS * NSTAGES : 1];

  const int h = static_cast<int>(blockIdx.x) % p.hkv;
  const int share_id = static_cast<int>(blockIdx.x) / p.hkv;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int G = p.group;

  // PAGED: tiles are TMA destinations with the 128-byte swizzle, which is a function of the
  // shared-memory address: the ring starts on a 1024-byte boundary.  A tile is HD/64 column
  // blocks of 16 rows x 128 bytes.
  const uint32_t smem_pad = PAGED ? ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u) : 0u;
  unsigned char* smem_al = smem_raw + smem_pad;
  const uint32_t ring = smem_u32(smem_al) + warp * (NSTAGES * 2 * TILE_BYTES);
  float* sm_o = reinterpret_cast<float*>(smem_al + NWARPS * NSTAGES * 2 * TILE_BYTES);  // [NWARPS][4][MROW]
  float* sm_m = sm_o + NWARPS * kDecodeMergeHeads * MROW;                              // [NWARPS][16]
  float* sm_l = sm_m + NWARPS * 16;                                                    // [NWARPS][16]
  auto toff = [](int row, int chunk) -> uint32_t {
    if constexpr (PAGED)
      return static_cast<uint32_t>((chunk >> 3) * (kDecodeGroupTokens * 128) + (row << 7) +
                                   (((chunk & 7) ^ (row & 7)) << 4));
    else
      return swz_offset<CH>(row, chunk);
  };
  if constexpr (PAGED) {
    if (threadIdx.x == 0) {
      for (int i = 0; i < NWARPS * NSTAGES; ++i) mbar_init(smem_u32(&s_bar[i]), 33);   // the lanes' copies + the byte count
      prefetch_tensormap(&tm_k);
      prefetch_tensormap(&tm_v);
      fence_mbar_init();
    }
  }
  // Behind its own K/V store the kernel starts early: it looks its share up and has the first groups
  // on their way (those without a row that the store writes) before the store is through.
  bool waited = false;
  auto wait_in_front = [&]() {
    if (waited) return;
    waited = true;
    grid_dependency_wait();
    grid_dependency_launch();
  };
  if (p.num_new < 0) wait_in_front();
  // the rows that the store writes, 32 of them a register
  constexpr int kNewRegs = kDecodeNewMax / 32;
  int fresh[kNewRegs];
#pragma unroll
  for (int i = 0; i < kNewRegs; ++i)
    fresh[i] = i * 32 + lane < p.num_new ? __ldg(after_wait(p.new_slots) + i * 32 + lane) : -1;
  const int32_t* indptr = after_wait(p.indptr);
  const int32_t* kv_lens = after_wait(p.kv_lens);

  // ---- sequences, 32 at a time in the lanes.  Positions are groups of 16 tokens; behind a
  // sequence's groups come `pad` empty positions, the price of the segment that ends there (a CTA
  // that holds the end of one sequence and the start of the next gets less to read).  A batch of few
  // sequences whose rounded-up pieces fit the GPU all the same is cut per sequence instead
  // (`aligned`): every CTA then has one segment.
  const int B = p.batch;
  int share = 0x7fffffff;
  float inv_share = 0.f;
  // n / share for n >= 0: the approximate quotient is off by one at most (quotients are below 2^20)
  auto over_share = [&](int n) -> int {
    int q = static_cast<int>(static_cast<float>(n) * inv_share);
    const int r = n - q * share;
    q += r < 0 ? -1 : r >= share ? 1 : 0;
    return q;
  };
  bool aligned = false;
  struct Window {        // 32 sequences from `base` on, in shared memory:
    int base;            // {first position, groups, first page / token of the index list, tokens}
    int4* at;
  };
  // tokens of sequence b (page-granular: clamped to what its pages hold), groups of them
  auto length = [&](int b, int& kvb, int& len) -> int {
    kvb = __ldg(indptr + b);
    const int64_t cap = static_cast<int64_t>(max(__ldg(indptr + b + 1) - kvb, 0)) * (PAGED ? p.page_size : 1);
    len = PAGED ? static_cast<int>(min(static_cast<int64_t>(max(__ldg(kv_lens + b), 0)), cap))
                : static_cast<int>(cap);
    return (len + kDecodeGroupTokens - 1) / kDecodeGroupTokens;
  };
  auto scan = [&](int x) -> int {   // inclusive, over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    return x;
  };
  auto padded = [&](int n) -> int { return n == 0 ? 0 : aligned ? (over_share(n - 1) + 1) * share : n + p.pad; };
  auto load_window = [&](Window& w, int base, int first) {
    int kvb = 0, len = 0;
    const int n = base + lane < B ? length(base + lane, kvb, len) : 0;
    const int room = padded(n);
    __syncwarp();
    w.base = base;
    w.at[lane] = make_int4(first + scan(room) - room, n, kvb, len);
    __syncwarp();
  };

  // ---- this CTA's share [r0, r1) of the positions, and the first sequence in it
  // (one window for the copies, which run ahead, one for the arithmetic)
  int4* windows = reinterpret_cast<int4*>(sm_l + NWARPS * 16) + warp * 64;
  Window pw{0, windows}, cw{0, windows + 32};
  int b0, b_stop = B, r0, r1;
  bool tail = true;           // no share behind this one: empty sequences at the end are this one's too
  if (p.num_shares == 0) {    // (scratch for one partial per sequence only: shares are whole sequences)
    b0 = share_id;
    b_stop = b0 + 1;
    load_window(pw, b0, 0);
    r0 = 0;
    r1 = 0x7fffffff;
  } else {
    // a lane sums a run of consecutive sequences; with at most 32 of them that is the window itself
    const int run = (B + 31) / 32;
    int sum = 0, n1 = 0, kvb1 = 0, len1 = 0, longest = 0;
    if (run == 1) {
      if (lane < B) n1 = length(lane, kvb1, len1);
      sum = padded(n1);
      longest = n1;
    } else {
      for (int j = 0; j < run; ++j) {
        int kvb, len;
        const int b = lane * run + j;
        if (b >= B) break;
        const int n = length(b, kvb, len);
        sum += padded(n);
        longest = max(longest, n);
      }
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    int total = __reduce_add_sync(0xffffffffu, sum);
    // whole waves of CTAs: 1.2 waves of equal shares take as long as two
    if (total <= p.wave * p.max_share || p.max_waves <= 1) {
      share = __float2int_ru(static_cast<float>(total) * p.inv_wave);     // (inv_wave is rounded up: one too many at most,
      share -= (share - 1) * p.wave >= total ? 1 : 0;                     // or too few of a total beyond 2^24, see below)
    } else {
      share = ceil_div(total, p.wave * min(ceil_div(total, p.wave * p.max_share), p.max_waves));
    }
    share = max(share, p.min_share);
    if (static_cast<int64_t>(share) * p.num_shares < total) share = ceil_div(total, p.num_shares);
    // The pieces of a sequence's head are merged by one warp, a row per piece.  Where there are many of them
    // the merge is as long as the loop and longer; share + longest / share * merge_row is least where the two
    // are equal.
    if (longest > p.max_pieces * share)
      share = max(share, static_cast<int>(fast_sqrt(static_cast<float>(longest) * p.merge_row)));
    share = (share + NWARPS - 1) / NWARPS * NWARPS;
    inv_share = __fdividef(1.f, static_cast<float>(share));
    if (run == 1) {
      const int pieces = n1 == 0 ? 0 : over_share(n1 - 1) + 1;
      aligned = __reduce_add_sync(0xffffffffu, pieces) <= min(p.wave, p.num_shares);
      if (aligned) {
        sum = pieces * share;
        total = __reduce_add_sync(0xffffffffu, sum);
      }
    }
    const int64_t start = static_cast<int64_t>(share_id) * share;
    if (start >= total && share_id > 0) return;
    r0 = static_cast<int>(start);
    tail = start + share >= total;
    r1 = tail ? total : r0 + share;
    // first sequence that starts at r0 or holds it
    const int incl = scan(sum);
    if (run == 1) {
      pw.at[lane] = make_int4(incl - sum, n1, kvb1, len1);
      const uint32_t m = __ballot_sync(0xffffffffu, lane < B && (incl - sum >= r0 || incl > r0));
      b0 = m != 0u ? __ffs(m) - 1 : B;
    } else {
      // in the first run that reaches r0, or right behind
      const int l = __ffs(__ballot_sync(0xffffffffu, incl >= r0)) - 1;
      int found = l * run + run, at = incl;    // (broadcast from lane l)
      if (lane == l) {
        int pos = incl - sum;
        for (int j = 0; j < run; ++j) {
          int kvb, len;
          const int b = l * run + j;
          if (b >= B) break;
          const int n = padded(length(b, kvb, len));
          if (pos >= r0 || pos + n > r0) {
            found = b;
            at = pos;
            break;
          }
          pos += n;
        }
      }
      b0 = __shfl_sync(0xffffffffu, found, l);
      at = __shfl_sync(0xffffffffu, at, l);
      load_window(pw, b0, at);
    }
  }
  __syncwarp();
  cw.base = pw.base;
  if (B <= 32) {
    cw.at = pw.at;             // (all sequences: neither moves on)
  } else {
    cw.at[lane] = pw.at[lane];
    __syncwarp();
  }
  if constexpr (PAGED) __syncthreads();     // the ring's barriers exist

  const unsigned char* __restrict__ kbase = static_cast<const unsigned char*>(p.k_cache);
  const unsigned char* __restrict__ vbase = static_cast<const unsigned char*>(p.v_cache);
  const int64_t slot_stride = static_cast<int64_t>(p.hkv) * ROW_BYTES;
  const int64_t head_off = static_cast<int64_t>(h) * ROW_BYTES;

  // ---- segment of a sequence
  struct Segment {
    int beg, end;        // positions of the whole sequence
    int t_lo, t_hi, ng;  // its tokens inside the share, groups of them
    int kvb, len;
  };
  auto segment = [&](Window& w, int b, Segment& s) -> bool {   // false: b is behind the share
    if (b >= b_stop) return false;
    if (b - w.base >= 32) {
      const int4 last = w.at[31];
      load_window(w, b, last.x + padded(last.y));
    }
    const int4 q4 = w.at[b - w.base];
    s.beg = q4.x;
    s.end = q4.x + q4.y;
    s.kvb = q4.z;
    s.len = q4.w;
    if (!tail && s.beg >= r1) return false;
    const int lo = max(s.beg, r0), hi = min(s.end, r1);
    s.t_lo = (lo - s.beg) * kDecodeGroupTokens;
    s.t_hi = min(s.len, (hi - s.beg) * kDecodeGroupTokens);
    s.ng = max(hi - lo, 0);
    return true;
  };

  // ---- the copies: this warp's groups of the share in order, round-robin among the warps.  The ids
  // of up to 32 of its groups (per-token form: the slots of two) come with one load, a lane each,
  // and the batch behind is on its way while one is used.
  constexpr int BATCH = PAGED ? 32 : 2;
  struct Batch {
    int count, t0, len;  // groups; token of the first one; tokens there are
    // PAGED: lane j, group j: first pool row, num_slots if the page is outside the pool (rows behind the pool
    // read as zeros); else lane 16 j + r: slot of row r, -1: zeros
    int y;
    uint32_t fresh;      // per-token form, before the wait
  };
  Segment ps;
  int pb = b0, pg = warp;
  bool more = segment(pw, pb, ps);
  auto load_batch = [&](Batch& w) {
    while (more && pg >= ps.ng) {
      pg -= ps.ng;
      more = segment(pw, ++pb, ps);
    }
    w.count = more ? min(BATCH, ceil_div(ps.ng - pg, NWARPS)) : 0;
    w.t0 = ps.t_lo + pg * kDecodeGroupTokens;
    w.len = PAGED ? ps.len : ps.t_hi;
    w.y = -1;
    pg += w.count * NWARPS;
    const int j = PAGED ? lane : lane / kDecodeGroupTokens;
    const int t = w.t0 + j * (NWARPS * kDecodeGroupTokens) + (PAGED ? 0 : lane % kDecodeGroupTokens);
    if (j < w.count && t < w.len) {
      // (pages of 16 tokens: no division)
      const int per = PAGED ? p.page_size : 1;
      const int page = PAGED && per != kDecodeGroupTokens ? t / per : PAGED ? t / kDecodeGroupTokens : t;
      const int id = __ldg(p.indices + ps.kvb + page);
      const int64_t row = static_cast<int64_t>(id) * per + (t - page * per);
      const int rows = PAGED ? min(kDecodeGroupTokens, w.len - t) : 1;
      if (id >= 0 && row + rows <= p.num_slots) w.y = static_cast<int>(row);
      else {                                        // page or slot outside the pool: zeros
        if (PAGED) w.y = static_cast<int>(p.num_slots);
        if (p.status) atomicExch(p.status, 2);
      }
    }
    if constexpr (!PAGED) {
      w.fresh = 0u;
      if (!waited) {       // lanes whose row the kernel in front writes
        bool hit = false;
#pragma unroll
        for (int i = 0; i < kNewRegs; ++i) {
          if (i * 32 >= p.num_new) break;
#pragma unroll 16
          for (int k = 0; k < 32; ++k) hit |= w.y == __shfl_sync(0xffffffffu, fresh[i], k);
        }
        w.fresh = __ballot_sync(0xffffffffu, hit && w.y >= 0);
      }
    }
  };
  auto bar_of = [&](int stage) { return smem_u32(&s_bar[PAGED ? warp * NSTAGES + stage : 0]); };
  Batch cur, nxt;
  cur.count = nxt.count = 0;
  int ck = 0;
  // copies of this warp's next group into a stage, if it has one
  auto issue_next = [&](int stage) {
    while (ck == cur.count) {
      if (nxt.count == 0 && !more) return;
      cur = nxt;
      ck = 0;
      load_batch(nxt);
    }
    if (!waited) {
      // does the group hold a row that the kernel in front writes?
      bool hit = false;
      if constexpr (PAGED) {
        const int y = __shfl_sync(0xffffffffu, cur.y, ck);
#pragma unroll
        for (int i = 0; i < kNewRegs; ++i) hit |= fresh[i] >= y && fresh[i] < y + kDecodeGroupTokens;
      } else {
        hit = (cur.fresh >> (ck * kDecodeGroupTokens) & 0xffffu) != 0u;
      }
      if (__any_sync(0xffffffffu, hit)) wait_in_front();
    }
    const uint32_t kdst = ring + stage * (2 * TILE_BYTES);
    const uint32_t vdst = kdst + TILE_BYTES;
    if constexpr (PAGED) {
      const uint32_t bar = bar_of(stage);
      const int y = __shfl_sync(0xffffffffu, cur.y, ck);
      const int n = min(kDecodeGroupTokens, cur.len - cur.t0 - ck * (NWARPS * kDecodeGroupTokens));
      if (n == kDecodeGroupTokens) {
        if (lane == 0) {
          mbar_arrive_expect_tx(bar, 2 * TILE_BYTES);
          tma_load_3d(kdst, &tm_k, 0, y, h * (HD / 64), bar);
          tma_load_3d(vdst, &tm_v, 0, y, h * (HD / 64), bar);
        }
      } else {
        // ragged last page of the sequence: valid rows by 16-byte copies, the rest zeros; the barrier
        // completes when the copies of all lanes have landed
#pragma unroll 4
        for (int k = 0; k < kDecodeGroupTokens * CH / 32; ++k) {
          const int e = k * 32 + lane;
          const int row = e / CH, chunk = e % CH;
          const bool ok = row < n && y < p.num_slots;
          const int64_t off =
              (ok ? static_cast<int64_t>(y + row) * slot_stride + head_off : 0) + chunk * 16;
          cp_async_16(kdst + toff(row, chunk), kbase + off, ok ? 16 : 0);
          cp_async_16(vdst + toff(row, chunk), vbase + off, ok ? 16 : 0);
        }
        if (lane == 0) mbar_arrive(bar);
      }
      cp_async_mbar_arrive(bar);
    } else {
      constexpr int ROWS_PER_PASS = 32 / CH == 0 ? 1 : 32 / CH;  // 2 at HD=128, 1 at HD=256
      constexpr int PASSES = kDecodeGroupTokens / ROWS_PER_PASS;
      const int chunk = lane % CH;
      const int rsub = lane / CH;
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        const int row = i * ROWS_PER_PASS + rsub;
        const int slot = __shfl_sync(0xffffffffu, cur.y, ck * kDecodeGroupTokens + row);
        const bool ok = slot >= 0;
        const int64_t off = (ok ? static_cast<int64_t>(slot) * slot_stride + head_off : 0) + chunk * 16;
        const uint32_t so = swz_offset<CH>(row, chunk);
        cp_async_16(kdst + so, kbase + off, ok ? 16 : 0);
        cp_async_16(vdst + so, vbase + off, ok ? 16 : 0);
      }
    }
    ++ck;
  };

  // ---- the arithmetic, segment by segment
  T* out = static_cast<T*>(p.out);
  constexpr int VPL = HD / 32, NV = VPL / 4;   // columns (16-byte pieces) of a row per lane
  bool alive = true;
  struct Partial {
    int b, first, count;     // sequence, its first share, its shares
  };
  Partial part0{0, 0, 0}, part1{0, 0, 0};   // the partial segments: part1 the latest, part0 the one before
  int pending = 0;
  int cg = warp;
  int stage = 0, fill = 0;          // ring position of this step / of the next copy
  int ahead = 0;                    // copies issued and not used yet
  uint32_t parity = 0;
  auto top_up = [&]() {             // every stage in flight
#pragma unroll 1
    for (; ahead < NSTAGES; ++ahead) {
      issue_next(fill);
      if constexpr (!PAGED) cp_async_commit();
      fill = fill + 1 == NSTAGES ? 0 : fill + 1;
    }
  };
  constexpr bool kQInSmem = HD == 256;
  unsigned char* sm_q = reinterpret_cast<unsigned char*>(sm_l + NWARPS * 16) + NWARPS * 64 * 16;
  Segment cs;
  for (int b = b0; segment(cw, b, cs); ++b) {
    if (PAGED && h == 0 && threadIdx.x == 0 && cs.beg >= r0 && p.status && __ldg(kv_lens + b) != cs.len)
      atomicExch(p.status, 2);   // a length that is negative or beyond the sequence's pages: clamped, reported
    if (cs.ng == 0 && cs.end > cs.beg) continue;   // (only its padding is in this share)
    // Q: fragments in registers (rows = query heads of this KV head, rows >= G are zero); at head_dim
    // 256, where they would spill, a swizzled tile in shared memory
    uint32_t qf[kQInSmem ? 1 : KSTEPS][4];
    bool q_loaded = kQInSmem;
    if constexpr (kQInSmem) {
      top_up();
      wait_in_front();
      const T* q = after_wait(static_cast<const T*>(p.q));
#pragma unroll
      for (int e = threadIdx.x; e < 16 * CH; e += NWARPS * 32) {
        const int row = e / CH, chunk = e % CH;
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (row < G)
          x = *reinterpret_cast<const uint4*>(q + (static_cast<int64_t>(b) * p.hq + static_cast<int64_t>(h) * G + row) * HD +
                                              chunk * 8);
        *reinterpret_cast<uint4*>(sm_q + swz_offset<CH>(row, chunk)) = x;
      }
      __syncthreads();
    }
    // (the gate's rows on their way into L2: they are wanted when the segment is merged)
    if (p.gate != nullptr && warp == 0) {
      const char* rows = reinterpret_cast<const char*>(static_cast<const T*>(p.gate) +
                                                       (static_cast<int64_t>(b) * p.hq + static_cast<int64_t>(h) * G) * HD);
      for (int c = lane * 128; c < G * ROW_BYTES; c += 32 * 128) prefetch_l2(rows + c);
    }
    float o[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;

    for (; cg < cs.ng; cg += NWARPS) {
      top_up();
      if (!kQInSmem && !q_loaded) {
        q_loaded = true;
        wait_in_front();
        const T* q = after_wait(static_cast<const T*>(p.q));
        {
          const int row = lane >> 2;
          const int c0 = (lane & 3) * 2;
          const uint32_t* q0 = reinterpret_cast<const uint32_t*>(
              q + (static_cast<int64_t>(b) * p.hq + static_cast<int64_t>(h) * G + row) * HD);
          const uint32_t* q1 = q0 + 8 * HD / 2;
          const bool v0 = row < G;
          const bool v1 = (row + 8) < G;
#pragma unroll
          for (int ks = 0; ks < KSTEPS; ++ks) {
            const int w = (ks * 16 + c0) >> 1;
            qf[ks][0] = v0 ? q0[w] : 0u;
            qf[ks][1] = v1 ? q1[w] : 0u;
            qf[ks][2] = v0 ? q0[w + 4] : 0u;
            qf[ks][3] = v1 ? q1[w + 4] : 0u;
          }
        }
      }
      if constexpr (PAGED) {
        // bounded wait for this step's stage
        const uint32_t bar = bar_of(stage);
        bool ok = !alive || mbar_try_wait(bar, parity);
        if (!ok) {
          const long long t0 = clock64();
          while (!(ok = mbar_try_wait(bar, parity)) && clock64() - t0 < kTcWaitCycles) {
          }
        }
        alive = __all_sync(0xffffffffu, alive && ok ? 1 : 0) != 0;
        if (!alive) continue;       // (gave up: the rest of the share is walked without its data)
      } else {
        cp_async_wait<NSTAGES - 1>();
        __syncwarp();
      }
      const uint32_t kt = ring + stage * (2 * TILE_BYTES);
      const uint32_t vt = kt + TILE_BYTES;

      // S = Q K^T for 16 tokens: two n-tiles of 8 tokens, each in two independent chains
      float s[2][4], s2[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[i][e] = s2[i][e] = 0.f;
      {
        const int mat = lane >> 3;
        const int row = (lane & 7) + ((mat >> 1) << 3);
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ks += 2) {
          uint32_t kf[4], kg[4];
          if constexpr (kQInSmem) {
            uint32_t qa[4], qb[4];
            ldmatrix_x4(qa, smem_u32(sm_q) + swz_offset<CH>(lane & 15, 2 * ks + (lane >> 4)));
            ldmatrix_x4(qb, smem_u32(sm_q) + swz_offset<CH>(lane & 15, 2 * ks + 2 + (lane >> 4)));
            ldmatrix_x4(kf, kt + toff(row, 2 * ks + (mat & 1)));
            ldmatrix_x4(kg, kt + toff(row, 2 * ks + 2 + (mat & 1)));
            MmaOp<T>::run(s[0], qa, kf[0], kf[1]);
            MmaOp<T>::run(s[1], qa, kf[2], kf[3]);
            MmaOp<T>::run(s2[0], qb, kg[0], kg[1]);
            MmaOp<T>::run(s2[1], qb, kg[2], kg[3]);
            continue;
          }
          ldmatrix_x4(kf, kt + toff(row, 2 * ks + (mat & 1)));
          ldmatrix_x4(kg, kt + toff(row, 2 * ks + 2 + (mat & 1)));
          MmaOp<T>::run(s[0], qf[ks], kf[0], kf[1]);
          MmaOp<T>::run(s[1], qf[ks], kf[2], kf[3]);
          MmaOp<T>::run(s2[0], qf[ks + 1], kg[0], kg[1]);
          MmaOp<T>::run(s2[1], qf[ks + 1], kg[2], kg[3]);
        }
      }
      // scale to base-2 logits, mask the tail of the range
      const int nvalid = cs.t_hi - cs.t_lo - cg * kDecodeGroupTokens;  // >= 1
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int col = nt * 8 + (lane & 3) * 2 + (e & 1);
          s[nt][e] = (col < nvalid) ? (s[nt][e] + s2[nt][e]) * p.scale_log2 : -INFINITY;
        }
      }
      const float mx0 = quad_max(fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1])));
      const float mx1 = quad_max(fmaxf(fmaxf(s[0][2], s[0][3]), fmaxf(s[1][2], s[1][3])));
      // the accumulator is rescaled only when some row's maximum has grown
      if (__any_sync(0xffffffffu, mx0 > m0 || mx1 > m1)) {
        const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);  // finite: column 0 is valid
        const float a0 = fast_exp2(m0 - mn0), a1 = fast_exp2(m1 - mn1);
        m0 = mn0;
        m1 = mn1;
        l0 *= a0;
        l1 *= a1;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          o[i][0] *= a0;
          o[i][1] *= a0;
          o[i][2] *= a1;
          o[i][3] *= a1;
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        s[nt][0] = fast_exp2(s[nt][0] - m0);
        s[nt][1] = fast_exp2(s[nt][1] - m0);
        s[nt][2] = fast_exp2(s[nt][2] - m1);
        s[nt][3] = fast_exp2(s[nt][3] - m1);
        l0 += s[nt][0] + s[nt][1];
        l1 += s[nt][2] + s[nt][3];
      }
      uint32_t pa[4];
      pa[0] = MmaOp<T>::pack(s[0][0], s[0][1]);
      pa[1] = MmaOp<T>::pack(s[0][2], s[0][3]);
      pa[2] = MmaOp<T>::pack(s[1][0], s[1][1]);
      pa[3] = MmaOp<T>::pack(s[1][2], s[1][3]);
      // O += P V
      {
        const int mat = lane >> 3;
        const int row = (lane & 7) + ((mat & 1) << 3);
#pragma unroll
        for (int j = 0; j < NT / 2; ++j) {
          uint32_t vf[4];
          ldmatrix_x4_trans(vf, vt + toff(row, 2 * j + (mat >> 1)));
          MmaOp<T>::run(o[2 * j], pa, vf[0], vf[1]);
          MmaOp<T>::run(o[2 * j + 1], pa, vf[2], vf[3]);
        }
      }
      __syncwarp();                 // every lane has read the stage: it is free
      --ahead;
      if (++stage == NSTAGES) {
        stage = 0;
        parity ^= 1;
      }
    }
    cg -= cs.ng;

    wait_in_front();     // (a warp without groups)
    // (a sequence's ragged last page came by ordinary copies, and its stage is filled by TMA next)
    if (PAGED && cs.t_hi % kDecodeGroupTokens != 0) fence_proxy_async_smem();
    // ---- end of the segment: the warps' partials are merged, four heads at a time, a warp per head
    // and a lane per VPL consecutive columns
    const bool whole = cs.beg >= r0 && cs.end <= r1;     // (positions of its groups, not of the padding)
    // (a share and a sequence boundary each open a new segment: share + sequence numbers them densely)
    const int64_t slot = (static_cast<int64_t>(share_id) + b) * p.hkv + h;
    l0 = quad_sum(l0);
    l1 = quad_sum(l1);
    if ((lane & 3) == 0) {
      sm_m[warp * 16 + (lane >> 2)] = m0;
      sm_m[warp * 16 + (lane >> 2) + 8] = m1;
      sm_l[warp * 16 + (lane >> 2)] = l0;
      sm_l[warp * 16 + (lane >> 2) + 8] = l1;
    }
    for (int gb = 0; gb < G; gb += kDecodeMergeHeads) {
      {
        // accumulator row of this lane inside the batch of heads: rows gb .. gb + 3 sit in the lower
        // (gb < 8) or upper half of the tile
        const int rr = (lane >> 2) - (gb & 7);
        if (rr >= 0 && rr < kDecodeMergeHeads) {
          float* ow = sm_o + (warp * kDecodeMergeHeads + rr) * MROW + (lane & 3) * 2;
          if (gb < 8) {
#pragma unroll
            for (int i = 0; i < NT; ++i) *reinterpret_cast<float2*>(ow + i * 8) = make_float2(o[i][0], o[i][1]);
          } else {
#pragma unroll
            for (int i = 0; i < NT; ++i) *reinterpret_cast<float2*>(ow + i * 8) = make_float2(o[i][2], o[i][3]);
          }
        }
      }
      const int g = gb + warp;
      const int64_t hq_idx = static_cast<int64_t>(b) * p.hq + static_cast<int64_t>(h) * G + g;
      GateVec<T, VPL> gate;
      if (g < G && whole) gate.load(static_cast<const T*>(p.gate), hq_idx * HD + lane * VPL);
      __syncthreads();
      if (g < G) {
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < NWARPS; ++w) M = fmaxf(M, sm_m[w * 16 + g]);
        float wgt[NWARPS];
        float den = 0.f;
#pragma unroll
        for (int w = 0; w < NWARPS; ++w) {
          wgt[w] = (M == -INFINITY) ? 0.f : fast_exp2(sm_m[w * 16 + g] - M);
          den += wgt[w] * sm_l[w * 16 + g];
        }
        float num[VPL];
#pragma unroll
        for (int e = 0; e < VPL; ++e) num[e] = 0.f;
#pragma unroll
        for (int w = 0; w < NWARPS; ++w) {
          const float4* row = reinterpret_cast<const float4*>(sm_o + (w * kDecodeMergeHeads + warp) * MROW + lane * VPL);
#pragma unroll
          for (int e4 = 0; e4 < NV; ++e4) {
            const float4 x = row[e4];
            num[4 * e4 + 0] += wgt[w] * x.x;
            num[4 * e4 + 1] += wgt[w] * x.y;
            num[4 * e4 + 2] += wgt[w] * x.z;
            num[4 * e4 + 3] += wgt[w] * x.w;
          }
        }
        if (whole) {
          const float inv = den > 0.f ? 1.f / den : 0.f;
#pragma unroll
          for (int e = 0; e < VPL; ++e) num[e] *= inv;
          write_decode_row<T, VPL>(out, gate, hq_idx * HD + lane * VPL, num);
        } else {
          float* row = p.part + (slot * G + g) * PROW;
#pragma unroll
          for (int e4 = 0; e4 < NV; ++e4)
            *reinterpret_cast<float4*>(row + lane * VPL + 4 * e4) =
                make_float4(num[4 * e4], num[4 * e4 + 1], num[4 * e4 + 2], num[4 * e4 + 3]);
          if (lane == 0) *reinterpret_cast<float2*>(row + HD) = make_float2(M, den);
        }
      }
      __syncthreads();   // the rows may be written again
    }
    if (!whole) {        // at most the first and the last segment of the share
      if (pending > 0) part0 = part1;
      part1.b = b;
      part1.first = over_share(cs.beg);
      part1.count = over_share(cs.end - 1) - part1.first + 1;
      ++pending;
    }
  }
  cp_async_wait<0>();

  // ---- the warp that arrives last at a (sequence, head)'s counter merges its partials:
  // out = sum_s 2^(M_s - M) O_s / sum_s 2^(M_s - M) l_s  (the second stage of the reference,
  // paged_decode_attention.metal:512-586, without a launch).  A warp arrives for the heads that it wrote, all
  // at once; per CTA instead (a barrier, one thread's arrivals, the pieces through shared memory) the tail of a
  // small call took 4.1 us, and a sequence's heads were all merged by one CTA.
  if (pending > 0) {
    const int mine = (G - warp + NWARPS - 1) / NWARPS;     // heads warp, warp + NWARPS, ... (none: <= 0)
    __syncwarp();
    bool last = false;
    if (lane < pending * 8 && (lane & 7) < mine) {         // (at most four heads: 16 / NWARPS)
      const Partial& part = lane < 8 ? part1 : part0;
      int* ticket = p.tickets + static_cast<int64_t>(part.b) * p.hq + h * G + warp + (lane & 7) * NWARPS;
      // the warp's partials are visible device-wide before the arrival, the others' after it
      last = atomic_add_acq_rel(ticket, 1) == part.count - 1;
      if (last) *ticket = 0;
    }
    uint32_t todo = __ballot_sync(0xffffffffu, last);
    __syncwarp();
#pragma unroll 1
    for (; todo != 0u; todo &= todo - 1) {
      const int l = __ffs(todo) - 1;
      const Partial& part = l < 8 ? part1 : part0;
      const int g = warp + (l & 7) * NWARPS;
      const int64_t oi = (static_cast<int64_t>(part.b) * p.hq + static_cast<int64_t>(h) * G + g) * HD + lane * VPL;
      GateVec<T, VPL> gate;
      gate.load(static_cast<const T*>(p.gate), oi);
      const float* rows = p.part + ((static_cast<int64_t>(part.first) + part.b) * p.hkv + h) * G * PROW + g * PROW;
      const int64_t pitch = static_cast<int64_t>(p.hkv) * G * PROW;     // from piece to piece
      float M = -INFINITY, den = 0.f, num[VPL];
#pragma unroll
      for (int e = 0; e < VPL; ++e) num[e] = 0.f;
      auto add_pieces = [&](auto fly) {
      constexpr int FLY = decltype(fly)::value;                         // pieces in flight
#pragma unroll 1
      for (int j0 = 0; j0 < part.count; j0 += FLY, rows += FLY * pitch) {
        const int m = min(FLY, part.count - j0);
        float4 x[FLY][NV];
        float2 ml = make_float2(-INFINITY, 0.f);                        // of piece lane % FLY
        if (lane % FLY < m) ml = __ldcg(reinterpret_cast<const float2*>(rows + (lane % FLY) * pitch + HD));
#pragma unroll
        for (int j = 0; j < FLY; ++j)
#pragma unroll
          for (int e4 = 0; e4 < NV; ++e4)
            x[j][e4] = j < m ? __ldcg(reinterpret_cast<const float4*>(rows + j * pitch + lane * VPL) + e4)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
        float mx = ml.x;
#pragma unroll
        for (int o2 = FLY / 2; o2 > 0; o2 >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o2));
        mx = fmaxf(mx, M);
        const float old = M == -INFINITY ? 0.f : fast_exp2(M - mx);
        const float w = ml.x == -INFINITY ? 0.f : fast_exp2(ml.x - mx);
        M = mx;
        float d = w * ml.y;
#pragma unroll
        for (int o2 = FLY / 2; o2 > 0; o2 >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o2);
        den = den * old + d;
#pragma unroll
        for (int e = 0; e < VPL; ++e) num[e] *= old;
#pragma unroll
        for (int j = 0; j < FLY; ++j) {
          const float wj = __shfl_sync(0xffffffffu, w, j);
#pragma unroll
          for (int e4 = 0; e4 < NV; ++e4) {
            num[4 * e4 + 0] += wj * x[j][e4].x;
            num[4 * e4 + 1] += wj * x[j][e4].y;
            num[4 * e4 + 2] += wj * x[j][e4].z;
            num[4 * e4 + 3] += wj * x[j][e4].w;
          }
        }
      }
      };
      // (16 pieces of a head are three reads of L2 in a row otherwise)
      if (part.count > 8) add_pieces(std::integral_constant<int, 16>{});
      else add_pieces(std::integral_constant<int, 8>{});
      const float inv = den > 0.f ? 1.f / den : 0.f;
#pragma unroll
      for (int e = 0; e < VPL; ++e) num[e] *= inv;
      write_decode_row<T, VPL>(out, gate, oi, num);
    }
  }
  if (!alive && p.status && lane == 0) atomicExch(p.status, 1);   // a wait ran out
}

}  // namespace msgl
