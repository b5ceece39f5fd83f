// Shared device helpers for the sm_100a paged-attention kernels: asynchronous
// 16-byte copies into shared memory, ldmatrix / mma.sync wrappers for the
// warp-level bf16/f16 tiles, the swizzled 256-byte-row shared-memory layout
// used for K/V token rows, and the base-2 online-softmax helpers.
#pragma once

#include <cuda.h>  // CUtensorMap (type only; no driver call is made from device code)
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace msgl {

constexpr float kLog2e = 1.4426950408889634f;

// ---------------------------------------------------------------- addresses
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// A K or V token row of one KV head is head_dim * 2 bytes = 16 chunks of 16
// bytes at head_dim 128.  Rows are stored 256 bytes apart; the 16-byte chunk
// index is XOR-ed with (row & 7) so that the eight rows an ldmatrix phase
// touches fall in eight different bank groups.
template <int kChunksPerRow>
__device__ __forceinline__ uint32_t swz_offset(int row, int chunk) {
  return static_cast<uint32_t>(row * (kChunksPerRow * 16) + ((chunk ^ (row & 7)) << 4));
}

// ---------------------------------------------------------------- cp.async
// 16-byte global -> shared copy that bypasses L1; src_bytes == 0 zero-fills.
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
               "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// All cp.async copies of this thread have landed.
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory");
}
// Counts an arrival: what the CTA wrote before (this thread is behind a CTA barrier) is visible to
// whoever sees the count, and what was written before the counts seen is visible here.
__device__ __forceinline__ int atomic_add_acq_rel(int* p, int v) {
  int old;
  asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

// ---------------------------------------------------------------- ldmatrix / mma
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

template <typename T>
struct MmaOp;
template <>
struct MmaOp<__nv_bfloat16> {
  __device__ __forceinline__ static void run(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  __device__ __forceinline__ static uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ __forceinline__ static __nv_bfloat16 from_float(float x) {
    return __float2bfloat16_rn(x);
  }
};
template <>
struct MmaOp<__half> {
  __device__ __forceinline__ static void run(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  __device__ __forceinline__ static uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ __forceinline__ static __half from_float(float x) { return __float2half_rn(x); }
};

// ---------------------------------------------------------------- misc
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
// (the same where the compiler may move it)
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed two-float arithmetic (one instruction for two lanes of a register pair).
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <typename T>
__device__ __forceinline__ float to_f32(T x);
template <>
__device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
template <>
__device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }

// out * sigmoid(gate) as the reference's layer computes it after the attention op
// (mini_sglang_mlx/models/qwen3_5.py:110): the attention output and the sigmoid are arrays of
// the 16-bit type, so each is rounded before the product is.
template <typename T>
__device__ __forceinline__ T apply_gate(float out, T gate) {
  const float o = to_f32(MmaOp<T>::from_float(out));
  // (a fast division, two units in the last place of fp32, in front of a rounding to 16 bits: the exact one
  // took most of a 128-row epilogue, 38 us at head_dim 256.  Below 2^-126 it gives zero.)
  const float s = to_f32(MmaOp<T>::from_float(__fdividef(1.f, 1.f + __expf(-to_f32(gate)))));
  return MmaOp<T>::from_float(o * s);
}

// Two elements of a row that is rounded already.  The product of two 16-bit numbers is exact in fp32, so one
// 16-bit multiplication rounds as apply_gate does.  (10 instructions a pair, 4 of them special-function, for 32.)
__device__ __forceinline__ uint32_t mul_pair(__nv_bfloat16, uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t mul_pair(__half, uint32_t a, uint32_t b) {
  const __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ float2 unpack_pair(__nv_bfloat16, uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
__device__ __forceinline__ float2 unpack_pair(__half, uint32_t v) { return __half22float2(*reinterpret_cast<__half2*>(&v)); }
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <typename T>
__device__ __forceinline__ uint32_t apply_gate_pair(uint32_t out, uint32_t gate) {
  const float2 g = unpack_pair(T{}, gate);
  float x0, x1;
  unpack_f32x2(mul_f32x2(pack_f32x2(g.x, g.y), pack_f32x2(-kLog2e, -kLog2e)), x0, x1);
  unpack_f32x2(add_f32x2(pack_f32x2(exp2_approx(x0), exp2_approx(x1)), pack_f32x2(1.f, 1.f)), x0, x1);
  return mul_pair(T{}, out, MmaOp<T>::pack(rcp_approx(x0), rcp_approx(x1)));
}

// Reduce over the four lanes that share a row of an m16n8 accumulator.
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
  return v;
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}

// Development aid, compiled in only with -DMSGL_TRACE: one record per CTA (SM, wall-clock entry
// and exit, cycle counts at the milestones of softmax group 0) read back through
// msgl_debug_read_cta_trace.
#ifdef MSGL_TRACE
constexpr int kTraceCtas = 8192;
__device__ long long g_cta_trace[kTraceCtas][32];
__device__ __forceinline__ long long trace_wall() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ int trace_smid() {
  int s;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(s));
  return s;
}
#define MSGL_TR(slot, value)                                                   \
  do {                                                                         \
    if (blockIdx.x < kTraceCtas) g_cta_trace[blockIdx.x][slot] = (value);      \
  } while (0)
#else
#define MSGL_TR(slot, value) do { } while (0)
#endif

// ---------------------------------------------------------------- mbarrier / TMA
constexpr long long kTcWaitCycles = 4000000000LL;            // bound of every barrier wait (~2 s)
constexpr int kTmaBoxRows = 16;   // token rows of one TMA box (= the smallest page)

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint32_t bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// CLUSTER: what was written before a release at cluster scope is visible once its count is seen (else:
// before a release of this CTA's threads).
template <bool CLUSTER = false>
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if constexpr (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok;
}
// Bounded wait: false after `limit` SM cycles or once another thread has given up.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_limit(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                long long limit) {
  if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
    if (*abort_flag != 0 || clock64() - t0 > limit) {
      *abort_flag = 1;
      return false;
    }
  }
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_wait_limit<CLUSTER>(bar, parity, abort_flag, kTcWaitCycles);
}
// Warp-uniform form: every lane waits, the warp agrees on the outcome, so that the
// warp-collective instructions that follow are executed by all lanes or by none.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity,
                                               volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait<CLUSTER>(bar, parity, abort_flag) ? 1 : 0) != 0;
}
// Arrive on `bar` once all cp.async copies issued so far by this thread have landed.
__device__ __forceinline__ void cp_async_mbar_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// One arrival that also announces `bytes` of bulk-copy traffic to come on this phase.
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
// TMA: box at element column x, row y of the 2-D tensor `tmap` into shared memory at dst; the
// bytes are counted on `bar` as they land.  Local memory only, one destination CTA.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tmap, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* tmap, int x, int y, int z,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
// Untiled bulk copies (16-byte aligned addresses, sizes a multiple of 16 bytes).
// shared -> global, tracked by the thread's bulk async-group:
__device__ __forceinline__ void bulk_store(void* gdst, uint32_t ssrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(ssrc),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// all bulk async-groups of this thread are complete (their writes have been performed)
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// orders this thread's accesses through the generic proxy with those of the async proxy
// (bulk copies), in every state space
__device__ __forceinline__ void fence_proxy_async_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Programmatic dependent launch.  The kernels of a layer (K/V store, norm + rotary + store, decode,
// prefill and its merge) are launched so that their CTAs may be resident while the kernel in front in
// the stream drains: they set up what is their own (shared memory, barriers, tensor memory), then
// grid_dependency_wait() blocks until the kernel in front has finished and its writes are visible
// (no-op when launched without the attribute).  A kernel lets the one behind it in
// (grid_dependency_launch) only after its own wait, so one that has started knows that everything but
// the kernel in front of it is complete.  That is what a layer call's attention builds on: the kernel in
// front is its own store, and everything older may be read before the wait.  In decode a CTA without
// work leaves without waiting; the first CTA of every head always waits, so the grid does.
// The kernels that make index arrays (metadata, gather, page expansion) are launched plainly: they start
// when everything in front is complete, and nothing starts before they are.
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// A pointer as it is known after the wait: no read through it moves in front of the wait, not even
// one that the compiler takes for a read of constant memory.
template <typename T>
__device__ __forceinline__ T* after_wait(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}
__device__ __forceinline__ void grid_dependency_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// One lane of a converged warp (the same lane every time for a full mask).
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .b32 rx;\n\t.reg .pred px;\n\t"
      "elect.sync rx|px, %1;\n\t"
      "@px mov.s32 %0, 1;\n\t}"
      : "+r"(pred)
      : "r"(0xFFFFFFFFu));
  return pred;
}

__host__ __device__ __forceinline__ int ceil_div(int a, int b) { return (a + b - 1) / b; }

}  // namespace msgl
