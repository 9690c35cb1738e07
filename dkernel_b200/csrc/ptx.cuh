// Thin wrappers over the sm_100a PTX this library uses: mbarrier, TMA
// (cp.async.bulk.tensor, each copy addressed to the issuing CTA only), tcgen05 (alloc / mma / commit / ld /
// st / fences) and the shared-memory / instruction descriptors of tcgen05.mma.
// Every wait is bounded: after kWaitLimitNs it gives up, records a status
// word and lets the kernel run to completion (results are then invalid and the
// host reports the status), so a protocol bug cannot hang the GPU.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "common.cuh"

namespace bsa {

// ------------------------------------------------------------------ host: TMA
// 4-D tiled tensor map over a (d, seq, head, batch) view of a strided tensor;
// strides in bytes must be multiples of 16 and the base 16-byte aligned.  The
// outer dimensions are stored in order of increasing stride; *_pos (1..3) say
// where each logical coordinate goes.
struct Tmap4 {
  CUtensorMap map;
  int seq_pos, head_pos, batch_pos;
  int head_bcast, batch_bcast;  // the dimension has extent 1 / stride 0: coordinate forced to 0
};
int make_tmap_4d(Tmap4* out, const void* base, int elem_bytes, uint64_t d, uint64_t seq,
                 uint64_t heads, uint64_t batch, int64_t seq_stride_b, int64_t head_stride_b,
                 int64_t batch_stride_b, uint32_t box_d, uint32_t box_seq, bool swizzle128,
                 bool is_bf16);

bool tma_compatible(const void* base, int elem_bytes, int64_t ss, int64_t sh, int64_t sb);

#if defined(__CUDACC__)
// ---------------------------------------------------------------- device side

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Arrival that publishes no memory writes of this thread (the consumer only needs to know that
// the thread has got that far): unlike the default release form it does not wait for the
// thread's global stores in flight.
__device__ __forceinline__ void mbar_arrive_relaxed(uint64_t* bar) {
  asm volatile("mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait.  mbarrier.try_wait suspends the thread in hardware for a while
// before it reports failure, so the loop neither burns issue slots nor adds
// wake-up latency; the bound is wall-clock time (kWaitLimitNs unless the caller
// gives its own).  Returns false when it gave up, after recording `code`:
// `status` points at the device status block {int code; int pad; int* mirror}.
// The first wait that gives up stores its code in the block and, when the host
// has registered one, in the host-visible mirror word, so that the host can
// notice without synchronising.
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s
static __device__ __noinline__ void record_wait_failure(int* status, int code) {
  if (!status) return;
  if (atomicCAS(status, 0, code) == 0) {
    int* mirror = *reinterpret_cast<int* volatile*>(status + 2);
    if (mirror) {
      *reinterpret_cast<volatile int*>(mirror) = code;
      __threadfence_system();
    }
  }
}
// Bounds-checking build (-DBSA_DEBUG_BOUNDS, `python -m dkernel_b200._build --debug`): the index
// invariants of the kernels are checked where the indices are formed.  A violated one records its
// code (800 + n) in the status block like a wait that gave up, and the access it guards is skipped:
// nothing traps, the context stays usable.  The release build compiles the checks away.
#ifdef BSA_DEBUG_BOUNDS
#define BSA_IN_BOUNDS(cond, status, code) ((cond) ? true : (::bsa::record_wait_failure((status), (code)), false))
#else
#define BSA_IN_BOUNDS(cond, status, code) (true)
#endif
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, int code,
                                          uint64_t limit_ns = kWaitLimitNs) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (global_timer_ns() - t0 > limit_ns) break;
  }
  record_wait_failure(status, code);
  return false;
}

// Weights 2^x as two 16-bit terms, p = hi + lo: hi cut off, lo what it leaves (rounded: 2^-16 of p or less).
// Where p > 0 both terms are, so that an infinity in V stays one (0 * inf would be NaN): lo is at least 2^-18 p in
// bf16.  f16 has no room for that below 1, so its x comes raised by kTermShift (2^15 at most when the reference
// maximum lags 2^8 behind), and lo is at least the smallest f16, 2^-31 of a weight at the reference.
// INF = false: V's type has no infinity.
template <bool BF16> constexpr float kTermShift = BF16 ? 0.f : 7.f;
template <bool BF16, bool INF>
__device__ __forceinline__ void two_terms(float p0, float p1, uint32_t& hi, uint32_t& lo) {
  float h0, h1;
  if (BF16) {
    asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(hi) : "r"(__float_as_uint(p0)), "r"(__float_as_uint(p1)));
    h0 = __uint_as_float(hi << 16);
    h1 = __uint_as_float(hi & 0xffff0000u);
    const __nv_bfloat162 l = __floats2bfloat162_rn(fmaxf(p0 - h0, p0 * 0x1p-18f), fmaxf(p1 - h1, p1 * 0x1p-18f));
    lo = *reinterpret_cast<const uint32_t*>(&l);
  } else {
    asm("cvt.rz.f16x2.f32 %0, %2, %1;" : "=r"(hi) : "f"(p0), "f"(p1));
    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    const __half2 l = __floats2half2_rn(INF && p0 > 0.f ? fmaxf(p0 - h.x, 0x1p-24f) : p0 - h.x,
                                        INF && p1 > 0.f ? fmaxf(p1 - h.y, 0x1p-24f) : p1 - h.y);
    lo = *reinterpret_cast<const uint32_t*>(&l);
  }
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// TMA tiled load, 4-D, into the issuing CTA's shared memory.
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0,
                                            int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
      "%5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// (d0, seq, head, batch) -> coordinates in the order the map stores them
__device__ __forceinline__ void tma_load_tile(void* dst, const Tmap4* tm, uint64_t* bar, int d0,
                                              int s, int h, int b) {
  if (tm->head_bcast) h = 0;
  if (tm->batch_bcast) b = 0;
  const int c1 = tm->seq_pos == 1 ? s : (tm->head_pos == 1 ? h : b);
  const int c2 = tm->seq_pos == 2 ? s : (tm->head_pos == 2 ? h : b);
  const int c3 = tm->seq_pos == 3 ? s : (tm->head_pos == 3 ? h : b);
  tma_load_4d(dst, &tm->map, bar, d0, c1, c2, c3);
}
// untiled bulk copy global -> shared (both addresses 16-byte aligned, bytes a multiple of 16)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// untiled bulk copy shared -> global (same alignment rules); completes with the thread's bulk groups
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ---- tcgen05 ----
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// All previously issued tcgen05.mma of this thread arrive on `bar` when done.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]
__device__ __forceinline__ void tc_mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Copy 128 rows x 32 bytes of a shared-memory matrix (described like an MMA
// operand) into 8 TMEM columns of all 128 lanes: exactly one k-step of a 16-bit
// A operand, in the layout tcgen05.mma expects for A in TMEM.  Ordered with the
// MMAs issued by the same thread.
__device__ __forceinline__ void tc_cp_128x256b(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::1.128x256b [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane
// (warp%4)*32 + t, v[i] = column i.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
        "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
      "%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
      "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
      "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
      "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
      "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
      : "memory");
}
// Packed fp32 pairs (sm_100): one instruction for two adjacent columns of a row.
__device__ __forceinline__ uint64_t f32x2(uint32_t lo_bits, uint32_t hi_bits) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo_bits), "r"(hi_bits));
  return r;
}
__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
  return f32x2(__float_as_uint(lo), __float_as_uint(hi));
}
__device__ __forceinline__ void f32x2_split(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor of tcgen05.mma for a 128-byte-swizzled tile
// whose 8-row groups are 1024 bytes apart (the layout TMA writes with
// CU_TENSOR_MAP_SWIZZLE_128B and a 128-byte inner box).
//   K-major  (rows = M/N index, 128 contiguous bytes = 64 K elements): SBO = 1024.
//   MN-major (rows = K index, 128 contiguous bytes = 64 M/N elements): SBO = 1024
//            between 8-row K groups, LBO = distance between 64-element M/N chunks.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr, uint32_t lbo_bytes,
                                                    uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)2 << 61;  // 128-byte swizzle
  return d;
}

// Descriptor of an un-swizzled tile made of core matrices of 8 rows x 16 bytes stored as 128
// contiguous bytes.  MN-major operand (a row = one K index, its 16 bytes = 8 M/N elements):
// lbo = distance between 8-row groups along K, sbo = between core matrices along M/N (the
// other way round than for the swizzled MN-major tile; established by test).
__device__ __forceinline__ uint64_t umma_desc_plain(uint32_t saddr, uint32_t lbo_bytes,
                                                    uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  return d;                // layout type 0: no swizzle
}

// Instruction descriptor of tcgen05.mma.kind::f16: fp32 accumulate, A/B of the
// same 16-bit type.
__device__ __forceinline__ uint32_t umma_idesc(bool bf16, int M, int N, bool a_mn_major,
                                               bool b_mn_major) {
  uint32_t d = 0;
  d |= 1u << 4;                    // D format: f32
  d |= (bf16 ? 1u : 0u) << 7;      // A format
  d |= (bf16 ? 1u : 0u) << 10;     // B format
  d |= (a_mn_major ? 1u : 0u) << 15;
  d |= (b_mn_major ? 1u : 0u) << 16;
  d |= (uint32_t)(N >> 3) << 17;
  d |= (uint32_t)(M >> 4) << 24;
  return d;
}
#endif  // __CUDACC__

}  // namespace bsa
