// Bandwidth-bound decode: one query token per sequence against contiguous K/V.
//
// Grid = (split, kv head x head group, sequence).  A CTA owns up to
// blocks_per_split attended blocks of one (sequence, kv head): one warp lists them, and
// their K and V tiles (TMA boxes of kTok tokens x D) stream through a 64 KB
// shared-memory ring (three CTAs fit per SM, so one CTA's prologue and epilogue
// are covered by the loads of the other two).  Every tile pair ("unit") belongs to ONE of the
// four consumer warps, so four units are worked on at a time and the fixed costs of a unit
// (barrier, maximum over the tokens, rescaling) are paid once per unit instead of once per warp.
// The products are transposed, S^T = K Q^T and O^T = V^T P^T, which puts the tokens (and the
// head dims) on the 16 rows of an m16n8k16 product and the q heads of the kv group on its 8
// columns: K/V are read from HBM once per group, and a group of four heads wastes half of a
// product instead of three quarters.
//
// Semantics follow the q_len == 1 case of
// dkernel/ops/sparse_attn_inference.py:503-514: positions are re-based to the
// first real token, the pattern row is (len - 1) / block_size, every real token
// of an attended block is visible.
#include <mutex>
#include <type_traits>

#include "ptx.cuh"

namespace bsa {

// Status block of the bounded waits: [0] code of the first wait that gave up (0 = none),
// [2..3] device-visible address of the host's mirror word (or null).
__device__ __align__(16) int g_wait_status[4] = {0, 0, 0, 0};

namespace {

constexpr int kRingBytes = 65536;        // K/V ring
constexpr int kMinCtas = 3;              // resident CTAs per SM the kernel is built for
constexpr int kConsumers = 4;            // consumer warps
constexpr int kDecThreads = 32 * (kConsumers + 1);
constexpr int kMaxTokens = 4096;         // tokens per CTA (a caller's blocks_per_split)
constexpr float kDecRescale = 8.0f;      // log2 of how far a maximum may grow before O is rescaled

constexpr int kClusterCtas = 128;        // CTAs per resident CTA of an SM up to which a grid runs as clusters
constexpr int kMaxCluster = 8;           // splits of a row that merge over distributed shared memory

// every thread of the cluster's CTAs; what was written to shared memory before is visible behind it
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// reads of another CTA's shared memory: the address that `p` has there
__device__ __forceinline__ uint32_t peer_smem(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float peer_load(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 peer_load4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

template <typename T> struct MmaType;
template <> struct MmaType<__half> {
  static __device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
};
template <> struct MmaType<__nv_bfloat16> {
  static __device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
};

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                        uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                          uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}

// transpose of an 8x8 tile of 16-bit elements held in fragment form (two elements per thread)
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(v));
  return d;
}
__device__ __forceinline__ float dec_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Shared-memory geometry.  16-bit K/V: a stage holds a K and a V tile as the tensor cores read
// them (D/64 sub-tiles of [kTok tokens][128 bytes], 128-byte swizzled).  8-bit (e4m3) K/V: a stage
// holds the two tiles as stored ([kTok tokens][D bytes]; 128-byte rows are swizzled, which keeps
// the V reads below free of bank conflicts); the consumer warps read the stored bytes with plain
// 16-byte loads and convert them straight into tensor-core fragments in registers.  e4m3 converts
// to f16 exactly and in one instruction per pair, so with an 8-bit cache the products run in f16
// whatever the type of q (q is converted once while it is staged; P lies in [0, 2^15]).
//
// Fragment trick of the 8-bit path: a product's contraction index may be enumerated in any order,
// and so may the output rows, as long as both operands (resp. the epilogue) agree.
//   K Q^T: thread (g, tq) of an m16n8k16 step holds k slots {2tq, 2tq+1, 8+2tq, 9+2tq}.  Over the
//          four steps of a 64-dim chunk these are made to stand for dims 16 tq .. 16 tq + 15 of the
//          chunk (step kk: dims 16 tq + 4 kk + {0,1} and + {2,3}), so a thread's share of a K row
//          is ONE 16-byte load and each of its four words converts into one step's A fragment.
//   V^T P^T: rows g and g + 8 of m-tile md stand for dims (D/8) g + 2 md and + 1, so thread g owns
//          D/8 consecutive dims: its share of a V row is one 16-byte (D = 128) load, and a byte
//          permute pairs the bytes of two token rows into the A fragment of an m-tile.
template <int D, bool FP8> struct DecGeo {
  static constexpr int kTok = D == 128 && !FP8 ? 32 : 64;   // tokens per unit
  static constexpr int kTileBytes = kTok * D * (FP8 ? 1 : 2);
  static constexpr int kStageBytes = 2 * kTileBytes;
  static constexpr int kStages = kRingBytes / kStageBytes;
  static constexpr bool kSwizzle = !FP8 || D == 128;
  static_assert(kStages % kConsumers == 0, "a stage belongs to one consumer warp");
  // byte offset of 16-byte chunk `chunk` of token row `tok` in a tile
  static __device__ __forceinline__ uint32_t off(int tok, int chunk) {
    if (FP8) return (uint32_t)(tok * D + ((kSwizzle ? chunk ^ (tok & 7) : chunk) << 4));
    return (uint32_t)((chunk >> 3) * (kTok * 128) + tok * 128 + (((chunk & 7) ^ (tok & 7)) << 4));
  }
};

template <int D, bool FP8, int NT> struct DecodeSmem {
  // after the 1024-aligned ring
  alignas(16) uint16_t q[NT * 8][D];           // q heads of the group, zero rows behind them
  uint64_t k_full[DecGeo<D, FP8>::kStages];
  uint64_t v_full[DecGeo<D, FP8>::kStages];
  float wm[kConsumers][NT * 8];
  float wl[kConsumers][NT * 8];
  int n_units;                                 // units of this CTA
  int2 unit[1];                                // first position of each unit and its place in the cache: max_units entries
};
template <int D, bool FP8, int NT> size_t dec_smem(int max_units) {
  return 1024 + kRingBytes + sizeof(DecodeSmem<D, FP8, NT>) + sizeof(int2) * (size_t)max_units;
}

// four e4m3 bytes of a word -> two f16x2: (byte 0, byte 1) and (byte 2, byte 3); exact
__device__ __forceinline__ void cvt_e4m3x4(uint32_t w, uint32_t& lo, uint32_t& hi) {
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\t"
      "cvt.rn.f16x2.e4m3x2 %0, a;\n\tcvt.rn.f16x2.e4m3x2 %1, b;\n\t}"
      : "=r"(lo), "=r"(hi) : "r"(w));
}
__device__ __forceinline__ uint32_t byte_perm(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// NT: 8-column tiles of q heads (heads_per_cta <= 8 NT).
//
// P enters V^T P^T as two 16-bit terms, P = hi + lo (two_terms), which keeps its fp32 value to 2^-16 (bf16) or better.
// One term rounds every weight at 2^-9 (bf16) or 2^-12 (f16), and a reference maximum that is raised lazily
// leaves not even a row's largest weights exact: error against 64 bits, apart from the rounding of the output,
// 1.53e-3 of the output with bf16 and 1.8e-4 with e4m3 K/V, now 4.6e-6 and 2.8e-7.  FOLD: where the last
// tile holds up to four heads, their lo terms take its columns 4..7 (its q rows 4..7 repeat rows 0..3, so that
// the logits are there already) and cost no product of their own (the e4m3 step below 53.0 instead of 55.7 us);
// those of a fuller tile are a second product on the same V fragments.
//
// Bound by HBM with a 16-bit cache; with an 8-bit cache by the fixed cost of a CTA (row lookup, first
// tiles, merge of the warps: 7 us) and the latency of a unit.  64 sequences of 1024..8192 tokens, 32/8
// heads, D 128, local 16 + stride 8, with the merge kernel: 68 us for the 401 MB of a bf16 cache, 53 us for
// the 203 MB of an e4m3 cache (67.5 and 52.4 with P in one term).  (78 and 79 us when all four warps shared a unit, 16 tokens each, with the
// heads on the rows; 71 and 56 us when a producer warp refilled K and V together after both were read.)
// Nine to 16 heads, 2 kv heads, D 128, the same sequences: 27 to 30 us bf16 (heads on the rows: 26 to 29),
// 29 to 31.5 e4m3 (30 to 32); D 64 18 to 19 us (19 to 21).
template <typename T, int D, bool FP8, int NT, bool FOLD>
__global__ void __launch_bounds__(kDecThreads, FP8 && D == 128 && NT == 2 ? 2 : kMinCtas)   // 2: spills otherwise
decode_kernel(const __grid_constant__ Tmap4 tmK, const __grid_constant__ Tmap4 tmV,
              bsa_decode_params p, int nsplit, int cl, int max_units, const int32_t* __restrict__ row_start,
              const int32_t* __restrict__ row_end, int* wait_status) {
  using Geo = DecGeo<D, FP8>;
  constexpr int kStages = Geo::kStages, kTok = Geo::kTok;
  constexpr int kLoTiles = FOLD ? NT - 1 : NT;   // column tiles whose lo terms are a product of their own
  constexpr int kTileBytes = Geo::kTileBytes;
  constexpr int kStageBytes = Geo::kStageBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint8_t* ring = smem;
  using MT = typename std::conditional<FP8, __half, T>::type;   // type of the tensor-core products
  constexpr bool kBf16 = std::is_same<MT, __nv_bfloat16>::value;
  constexpr float kShift = kTermShift<kBf16>;
  auto* sm = reinterpret_cast<DecodeSmem<D, FP8, NT>*>(smem + kRingBytes);

  // the merge kernel behind this one may be made resident as soon as every CTA got here
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // non-zero: an earlier wait gave up.  Looked at after the row lookup, whose chain of dependent loads
  // (ranges, row pointer, columns) is what a CTA begins with: no need to put this load in front of it.
  const int gave_up = *reinterpret_cast<volatile int*>(wait_status);
  const int sp = blockIdx.x, b = blockIdx.z;
  // Row of q, o and lse: the sequence's number, or (packed batch of chunks and decode tokens) the
  // row of its single query token; sequences with another number of query tokens are not served here.
  // That launch is a programmatic dependent of the prefill kernel, of which it reads nothing; its first
  // CTA does not leave before that grid has completed, so that what follows in the stream follows both.
  // The others leave when they are done: waiting, they would hold the places of rows still to be worked on
  // (24 chunks of 64 tokens + 8 decode tokens: 106 -> 92 us; 7 chunks + 1 token: 43.7 -> 34 us).
  const auto leave = [&] {
    if (row_start && blockIdx.x + blockIdx.y + blockIdx.z == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  };
  int qb = b;
  if (row_start) {
    qb = row_start[b];
    if (row_end[b] - qb != 1) { leave(); return; }
  }
  const int G = p.hq / p.hkv;
  const int GH = p.heads_per_cta;
  const int groups_per_kv = G / GH;
  const int kvh = blockIdx.y / groups_per_kv;
  const int h0 = kvh * G + (blockIdx.y % groups_per_kv) * GH;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bs = p.block_size;
  const bool q_vec = reinterpret_cast<uintptr_t>(p.q) % 16 == 0 && p.q_sb % 8 == 0 && p.q_sh % 8 == 0;
  // e4m3 K carries a per-tensor scale: it folds into the logit scale (V's goes on the output)
  const float scale2 = p.sm_scale * kLog2e * (FP8 ? p.k_scale : 1.f);

  const int ks = p.k_start ? p.k_start[b] : 0;
  const int ke = p.k_end ? p.k_end[b] : p.sk;
  const int local_len = ke - ks;
  const int pos0 = p.k_pos0 ? p.k_pos0[b] : 0;
  const int total = p.k_total ? p.k_total[b] : pos0 + local_len;
  const int end_pos = p.k_blk_mod > 1 ? total : min(total, pos0 + local_len);

  // A KV shard is either a contiguous position range [pos0, pos0 + stored) or, with k_blk_mod = W
  // > 1, the blocks whose index is congruent to k_blk_rem modulo W, stored back to back (block c
  // of the sequence is local block c / W).
  const int mod = p.k_blk_mod > 1 ? p.k_blk_mod : 1;
  auto load_tile = [&](int u, bool is_v) {
    const int s = u % kStages;
    uint64_t* bar = is_v ? &sm->v_full[s] : &sm->k_full[s];
    mbar_expect_tx(bar, kTileBytes);
    const int tok = sm->unit[u].y;
    // a unit starts inside the stored tokens of its kv head (its tail may be past them)
    (void)BSA_IN_BOUNDS(tok >= 0 && tok < p.sk && kvh >= 0 && kvh < p.hkv && b < p.batch, wait_status, 821);
    uint8_t* dst = ring + s * kStageBytes + (is_v ? kTileBytes : 0);
    const Tmap4* tm = is_v ? &tmV : &tmK;
    // 8-bit: one box of [kTok tokens][D bytes], as stored
    constexpr int kBoxes = FP8 ? 1 : D / 64;
#pragma unroll
    for (int c = 0; c < kBoxes; ++c) tma_load_tile(dst + c * (kTok * 128), tm, bar, c * 64, tok, kvh, b);
  };

  if (warp == kConsumers) {
    if (lane == 0) tma_prefetch_desc(&tmK.map);
    if (lane == 1) tma_prefetch_desc(&tmV.map);
    // ---- this warp finds the attended blocks of this CTA: the sp-th group of
    // blocks_per_split row entries that lie in the shard.  The row is read 32 entries at a time
    // (one coalesced load and one vote per chunk instead of a chain of dependent loads), and the
    // first tiles are requested before the rest of the CTA has staged Q.
    int nu = 0;
    if (total > 0 && local_len > 0) {
      const int row = (total - 1) / bs;
      const int hp = pattern_head(h0, p.h_pat, p.hq, p.hkv);
      int c_beg = 0, c_end = 0;
      if (row < p.n_rows) {
        const int32_t* cr = p.crow + (int64_t)hp * p.crow_sh;
        c_beg = __ldg(cr + row);
        c_end = __ldg(cr + row + 1);
      }
      const int32_t* cols = p.col + (int64_t)hp * p.col_sh;
      const int subs = bs / kTok;
      // a cluster's CTAs take the entries in turns, which keeps their shares of any row level
      const int want0 = cl > 1 ? 0 : sp * p.blocks_per_split, want1 = want0 + cl * p.blocks_per_split;
      int seen = 0;   // row entries of the shard met so far
      for (int e0 = c_beg; e0 < c_end && seen < want1; e0 += 32) {
        const int e = e0 + lane;
        const int c = e < c_end ? __ldg(cols + e) : -1;
        const bool mine = c >= 0 && (mod == 1 ? c * bs >= pos0 : c % mod == p.k_blk_rem);
        const uint32_t vote = __ballot_sync(0xffffffffu, mine);
        const int idx = seen + __popc(vote & ((1u << lane) - 1u));
        int valid_units = 0;
        if (mine && idx >= want0 && idx < want1 && (cl == 1 || idx % cl == sp)) {
          for (int s = 0; s < subs; ++s) {
            // positions grow with the entry index, so the units past the end form a tail
            const int pos = c * bs + s * kTok;
            const int u = (idx - want0) / cl * subs + s;
            if (pos < end_pos && u < max_units) {
              sm->unit[u] = make_int2(pos, mod == 1 ? ks + (pos - pos0) : ks + (c / mod) * bs + s * kTok);
              ++valid_units;
            }
          }
        }
        nu += __reduce_add_sync(0xffffffffu, valid_units);
        seen += __popc(vote);
      }
    }
    if (gave_up) nu = cl > 1 ? 0 : -1;   // no CTA of a cluster leaves before the others have read its part
    __syncwarp();
    if (lane == 0) {
      sm->n_units = nu;
      for (int s = 0; s < kStages; ++s) {
        mbar_init(&sm->k_full[s], 1);
        mbar_init(&sm->v_full[s], 1);
      }
      mbar_fence_init();
      for (int u = 0; u < nu && u < kStages; ++u) load_tile(u, false);
      for (int u = 0; u < nu && u < kStages; ++u) load_tile(u, true);
    }
  } else {
    // q heads of the group -> rows of the q tile (rows of no head are zero), 16 bytes a thread.  The maximum is
    // taken and the end of the sequence masked before the logits are scaled, which asks for a positive
    // scale: a negative one hands its sign to q here, and scale 0 makes the products themselves zero.
    for (int i = tid; i < NT * 8 * D / 8; i += kConsumers * 32) {
      const int row = i / (D / 8), c = i % (D / 8);
      const int r = FOLD && row >= NT * 8 - 4 ? row - 4 : row;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < GH) {
        const T* src = reinterpret_cast<const T*>(p.q) + (int64_t)qb * p.q_sb + (int64_t)(h0 + r) * p.q_sh + c * 8;
        if (q_vec) {
          v = *reinterpret_cast<const uint4*>(src);
        } else {
          alignas(16) T tmp[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) tmp[e] = src[e];
          v = *reinterpret_cast<const uint4*>(tmp);
        }
        if (!(scale2 > 0.f)) {
          T* e = reinterpret_cast<T*>(&v);
#pragma unroll
          for (int j = 0; j < 8; ++j) e[j] = Elem<T>::from_f(Elem<T>::to_f(e[j]) * (scale2 < 0.f ? -1.f : scale2));
        }
        if (!std::is_same<MT, T>::value) {   // bf16 queries against an 8-bit cache: products run in f16
          const T* e = reinterpret_cast<const T*>(&v);
          alignas(16) __half hq[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) hq[j] = __float2half_rn(fminf(fmaxf(Elem<T>::to_f(e[j]), -65504.f), 65504.f));
          v = *reinterpret_cast<const uint4*>(hq);
        }
      }
      reinterpret_cast<uint4*>(&sm->q[0][0])[i] = v;
    }
  }
  __syncthreads();
  const int n_units = sm->n_units;
  if (n_units < 0) { leave(); return; }   // outputs are undefined until the host has cleared the status
  // one split and an output tensor: write the final rows; otherwise an fp32 partial per split
  const bool final_out = nsplit == 1 && p.o != nullptr;

  if (n_units == 0 && cl == 1) {  // nothing attended here: an empty partial (uniform exit)
    for (int i = tid; i < GH * D; i += kDecThreads) {
      const int h = h0 + i / D, d = i % D;
      if (final_out) {
        reinterpret_cast<T*>(p.o)[(int64_t)qb * p.o_sb + (int64_t)h * p.o_sh + d] = Elem<T>::from_f(0.f);
      } else {
        p.ws[(((int64_t)b * p.hq + h) * nsplit + sp) * D + d] = 0.f;
      }
    }
    for (int i = tid; i < GH; i += kDecThreads) {
      const int h = h0 + i;
      if (final_out) {
        if (p.lse) p.lse[(int64_t)qb * p.lse_sb + (int64_t)h * p.lse_sh] = -INFINITY;
      } else {
        p.ws[(int64_t)p.batch * p.hq * nsplit * D + ((int64_t)b * p.hq + h) * nsplit + sp] = -INFINITY;
      }
    }
    leave();
    return;
  }

  const int g = lane >> 2, tq = lane & 3;
  float oacc[D / 16][NT][4];   // O^T: rows = dims, columns = heads
#pragma unroll
  for (int i = 0; i < D / 16; ++i)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) oacc[i][nt][0] = oacc[i][nt][1] = oacc[i][nt][2] = oacc[i][nt][3] = 0.f;

  if (warp < kConsumers) {
    // ------------------------------------------------------------ consumers
    // A stage belongs to one warp, which asks for the next tile itself: K's place is refilled while the
    // softmax and V^T P^T of the unit are computed, V's while the next unit's K Q^T is.
    uint32_t qb[D / 16][NT][2];   // Q^T as the B operand: column n = g is head 8 nt + g
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint32_t* q32 = reinterpret_cast<const uint32_t*>(sm->q[nt * 8 + g]);
        // k slots (2tq, 2tq+1) and (8+2tq, 9+2tq) of step kk: the dims of the same numbers, or
        // (8-bit K/V) dims 16 tq + 4 (kk % 4) + {0,1} / {2,3} of 64-dim chunk kk / 4
        const int d0 = FP8 ? (kk >> 2) * 64 + tq * 16 + (kk & 3) * 4 : kk * 16 + tq * 2;
        const int d1 = FP8 ? d0 + 2 : d0 + 8;
        qb[kk][nt][0] = q32[d0 >> 1];
        qb[kk][nt][1] = q32[d1 >> 1];
      }
    // per head 8 nt + 2 tq + e: reference maximum (log2 domain), this thread's share of the sum
    float m[NT][2], l[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) { m[nt][0] = m[nt][1] = -INFINITY; l[nt][0] = l[nt][1] = 0.f; }
    const float mul = scale2 == 0.f ? 1.f : fabsf(scale2);   // q carries the sign
    const uint32_t ring_u32 = smem_u32(ring);

    for (int u = warp; u < n_units; u += kConsumers) {
      const int s = u % kStages;
      const uint32_t ph = (u / kStages) & 1;
      if (!mbar_wait(&sm->k_full[s], ph, wait_status, 102)) break;
      const uint32_t kbase = ring_u32 + s * kStageBytes;
      const uint32_t vbase = kbase + kTileBytes;
      const uint8_t* k8 = ring + s * kStageBytes;    // the tiles as generic pointers (8-bit path)
      const uint8_t* v8 = k8 + kTileBytes;
      const int valid = end_pos - sm->unit[u].x;   // tokens of this unit that exist (may exceed kTok)
      // S^T = K Q^T
      float sacc[kTok / 16][NT][4];
#pragma unroll
      for (int mt = 0; mt < kTok / 16; ++mt) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) sacc[mt][nt][0] = sacc[mt][nt][1] = sacc[mt][nt][2] = sacc[mt][nt][3] = 0.f;
        if (FP8) {
#pragma unroll
          for (int c = 0; c < D / 64; ++c) {
            const uint4 lo = *reinterpret_cast<const uint4*>(k8 + Geo::off(mt * 16 + g, c * 4 + tq));
            const uint4 hi = *reinterpret_cast<const uint4*>(k8 + Geo::off(mt * 16 + g + 8, c * 4 + tq));
            const uint32_t wl[4] = {lo.x, lo.y, lo.z, lo.w}, wh[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              uint32_t a[4];
              cvt_e4m3x4(wl[kk], a[0], a[2]);
              cvt_e4m3x4(wh[kk], a[1], a[3]);
#pragma unroll
              for (int nt = 0; nt < NT; ++nt)
                MmaType<MT>::mma(sacc[mt][nt], a, qb[c * 4 + kk][nt][0], qb[c * 4 + kk][nt][1]);
            }
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            uint32_t a[4];
            ldsm_x4(kbase + Geo::off(mt * 16 + (lane & 15), kk * 2 + (lane >> 4)), a[0], a[1], a[2], a[3]);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) MmaType<MT>::mma(sacc[mt][nt], a, qb[kk][nt][0], qb[kk][nt][1]);
          }
        }
      }
      __syncwarp();   // every lane has read K
      if (lane == 0 && u + kStages < n_units) load_tile(u + kStages, false);
      // mask; per head: maximum over the unit's tokens, reference maximum, sum
      float alpha[NT][2];
      bool need = false;
      if (valid < kTok) {
#pragma unroll
        for (int mt = 0; mt < kTok / 16; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (mt * 16 + g + (e >> 1) * 8 >= valid) sacc[mt][nt][e] = -INFINITY;
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float mx = -INFINITY;
#pragma unroll
          for (int mt = 0; mt < kTok / 16; ++mt) mx = fmaxf(mx, fmaxf(sacc[mt][nt][e], sacc[mt][nt][2 + e]));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
          mx *= mul;
          alpha[nt][e] = 1.f;
          if (m[nt][e] == -INFINITY) {
            m[nt][e] = mx;         // nothing summed so far
          } else if (mx > m[nt][e] + kDecRescale) {
            alpha[nt][e] = dec_ex2(m[nt][e] - mx);
            m[nt][e] = mx;
            need = true;
          }
        }
      if (__any_sync(0xffffffffu, need)) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          l[nt][0] *= alpha[nt][0];
          l[nt][1] *= alpha[nt][1];
#pragma unroll
          for (int i = 0; i < D / 16; ++i) {
            oacc[i][nt][0] *= alpha[nt][0]; oacc[i][nt][1] *= alpha[nt][1];
            oacc[i][nt][2] *= alpha[nt][0]; oacc[i][nt][3] *= alpha[nt][1];
          }
        }
      }
      // P^T as the B operand: the 8x8 tiles of S^T's accumulator layout, transposed; FOLD: lo in columns 4..7 of the last tile
      uint32_t pb[kTok / 16][NT][2], pl[kTok / 16][NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const float n0 = m[nt][0] == -INFINITY ? 0.f : kShift == 0.f ? -m[nt][0] : kShift - m[nt][0];
        const float n1 = m[nt][1] == -INFINITY ? 0.f : kShift == 0.f ? -m[nt][1] : kShift - m[nt][1];
#pragma unroll
        for (int mt = 0; mt < kTok / 16; ++mt) {
          const float p0 = dec_ex2(fmaf(sacc[mt][nt][0], mul, n0)), p1 = dec_ex2(fmaf(sacc[mt][nt][1], mul, n1));
          const float p2 = dec_ex2(fmaf(sacc[mt][nt][2], mul, n0)), p3 = dec_ex2(fmaf(sacc[mt][nt][3], mul, n1));
          l[nt][0] += p0 + p2;
          l[nt][1] += p1 + p3;
          uint32_t hi0, lo0, hi1, lo1;
          two_terms<kBf16, !FP8>(p0, p1, hi0, lo0);
          two_terms<kBf16, !FP8>(p2, p3, hi1, lo1);
          pb[mt][nt][0] = transpose8x8(FOLD && nt == NT - 1 && tq >= 2 ? lo0 : hi0);
          pb[mt][nt][1] = transpose8x8(FOLD && nt == NT - 1 && tq >= 2 ? lo1 : hi1);
          if (nt < kLoTiles) {
            pl[mt][nt][0] = transpose8x8(lo0);
            pl[mt][nt][1] = transpose8x8(lo1);
          }
        }
      }
      if (!mbar_wait(&sm->v_full[s], ph, wait_status, 101)) break;
      if (!FP8 && valid < kTok) {
        // rows past the end of the sequence may hold anything: clear them in V so that 0 * garbage
        // cannot produce NaN (the 8-bit path replaces them as it reads V)
        uint8_t* vgen = ring + s * kStageBytes + kTileBytes;
        for (int t = valid; t < kTok; ++t)
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            reinterpret_cast<uint32_t*>(vgen + c * (kTok * 128) + t * 128)[lane] = 0u;
        fence_proxy_async();  // order these writes before the next TMA into the stage
        __syncwarp();
      }
      // O^T += V^T P^T
#pragma unroll
      for (int mt = 0; mt < kTok / 16; ++mt) {
        if (FP8) {
          // k slots (2tq, 2tq+1, 8+2tq, 9+2tq) are the token rows of the same numbers; the thread's
          // D/8 consecutive dims of each row arrive in one load (zero past the sequence end)
          constexpr int kDims = D / 8;
          uint32_t rows[4][kDims / 4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int tok = mt * 16 + (i >> 1) * 8 + tq * 2 + (i & 1);
            if (kDims == 16) {
              const uint4 r = tok < valid ? *reinterpret_cast<const uint4*>(v8 + Geo::off(tok, g))
                                          : make_uint4(0u, 0u, 0u, 0u);
              rows[i][0] = r.x; rows[i][1] = r.y; rows[i][kDims / 4 - 2] = r.z; rows[i][kDims / 4 - 1] = r.w;
            } else {
              const uint2 r = tok < valid ? *reinterpret_cast<const uint2*>(v8 + tok * D + g * kDims)
                                          : make_uint2(0u, 0u);
              rows[i][0] = r.x; rows[i][kDims / 4 - 1] = r.y;
            }
          }
#pragma unroll
          for (int md = 0; md < D / 16; ++md) {
            const int wi = md >> 1;
            const uint32_t sel = (md & 1) ? 0x7362u : 0x5140u;   // {a.b, b.b, a.b+1, b.b+1}, b = 0 or 2
            uint32_t a[4];
            cvt_e4m3x4(byte_perm(rows[0][wi], rows[1][wi], sel), a[0], a[1]);   // tokens 2tq, 2tq+1
            cvt_e4m3x4(byte_perm(rows[2][wi], rows[3][wi], sel), a[2], a[3]);   // tokens 8+2tq, 9+2tq
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) MmaType<MT>::mma(oacc[md][nt], a, pb[mt][nt][0], pb[mt][nt][1]);
#pragma unroll
            for (int nt = 0; nt < kLoTiles; ++nt) MmaType<MT>::mma(oacc[md][nt], a, pl[mt][nt][0], pl[mt][nt][1]);
          }
        } else {
#pragma unroll
          for (int md = 0; md < D / 16; ++md) {
            const int j = lane >> 3;
            uint32_t a[4];
            ldsm_x4_t(vbase + Geo::off(mt * 16 + (j >> 1) * 8 + (lane & 7), md * 2 + (j & 1)), a[0], a[1], a[2], a[3]);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) MmaType<MT>::mma(oacc[md][nt], a, pb[mt][nt][0], pb[mt][nt][1]);
#pragma unroll
            for (int nt = 0; nt < kLoTiles; ++nt) MmaType<MT>::mma(oacc[md][nt], a, pl[mt][nt][0], pl[mt][nt][1]);
          }
        }
      }
      __syncwarp();   // every lane has read V
      if (lane == 0 && u + kStages < n_units) load_tile(u + kStages, true);
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) l[nt][e] += __shfl_xor_sync(0xffffffffu, l[nt][e], o);
        if (g == 0) {
          sm->wm[warp][nt * 8 + 2 * tq + e] = m[nt][e] - kShift;   // the maximum that O and l are relative to
          sm->wl[warp][nt * 8 + 2 * tq + e] = l[nt][e];
        }
      }
  }
  __syncthreads();  // every tile has been consumed: the ring is free
  // partial outputs, [warp][head][D]; four floats of padding per row spread the writes over the banks
  constexpr int kRow = D + 4;
  float* Om = reinterpret_cast<float*>(ring);
  static_assert(kConsumers * NT * 8 * kRow * 4 <= kRingBytes, "partial outputs must fit the ring");
  if (warp < kConsumers) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float* h_lo = Om + (warp * NT * 8 + nt * 8 + 2 * tq) * kRow;   // heads 2tq and 2tq + 1
      float* h_hi = h_lo + kRow;
#pragma unroll
      for (int md = 0; md < D / 16; ++md) {
        // rows g and g + 8 of m-tile md: the dims of the same numbers, or (8-bit K/V) two neighbours
        const int d0 = FP8 ? (D / 8) * g + 2 * md : md * 16 + g;
        const int d1 = FP8 ? d0 + 1 : d0 + 8;
        h_lo[d0] = oacc[md][nt][0]; h_hi[d0] = oacc[md][nt][1];
        h_lo[d1] = oacc[md][nt][2]; h_hi[d1] = oacc[md][nt][3];
      }
    }
  }
  __syncthreads();  // partial outputs are in shared memory

  const bool o_vec = reinterpret_cast<uintptr_t>(p.o) % 8 == 0 && p.o_sb % 4 == 0 && p.o_sh % 4 == 0;
  const bool ws_vec = reinterpret_cast<uintptr_t>(p.ws) % 16 == 0;
  auto store = [&](int r, int d, float4 acc, float mf, float l) {
    const float inv = (l > 0.f ? 1.f / l : 0.f) * (FP8 ? p.v_scale : 1.f);   // e4m3 V: per-tensor scale
    const float lse = l > 0.f ? (mf + log2f(l)) * kLn2 : -INFINITY;
    acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
    const int h = h0 + r;
    if (final_out) {
      T* dst = reinterpret_cast<T*>(p.o) + (int64_t)qb * p.o_sb + (int64_t)h * p.o_sh + d;
      if (o_vec) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(MmaType<T>::pack(acc.x, acc.y), MmaType<T>::pack(acc.z, acc.w));
      } else {
        dst[0] = Elem<T>::from_f(acc.x); dst[1] = Elem<T>::from_f(acc.y);
        dst[2] = Elem<T>::from_f(acc.z); dst[3] = Elem<T>::from_f(acc.w);
      }
      if (d == 0 && p.lse) p.lse[(int64_t)qb * p.lse_sb + (int64_t)h * p.lse_sh] = lse;
    } else {
      if (BSA_IN_BOUNDS(h < p.hq && sp < nsplit && d < D, wait_status, 822)) {
        float* dst = p.ws + (((int64_t)b * p.hq + h) * nsplit + sp) * D + d;
        if (ws_vec) *reinterpret_cast<float4*>(dst) = acc;
        else { dst[0] = acc.x; dst[1] = acc.y; dst[2] = acc.z; dst[3] = acc.w; }
      }
      if (d == 0)
        p.ws[(int64_t)p.batch * p.hq * nsplit * D + ((int64_t)b * p.hq + h) * nsplit + sp] = lse;
    }
  };
  // this CTA's part of a cluster's row: sums relative to the CTA's own maximum, behind the warps' parts
  float* part = Om + kConsumers * NT * 8 * kRow;   // [NT * 8][D], then the maxima and the sums
  float* part_m = part + NT * 8 * D;
  float* part_l = part_m + NT * 8;
  static_assert((kConsumers * NT * 8 * kRow + NT * 8 * (D + 2)) * 4 <= kRingBytes, "both must fit the ring");
  for (int i = tid; i < GH * (D / 4); i += kDecThreads) {
    const int r = i / (D / 4), d = i % (D / 4) * 4;
    float mf = -INFINITY;
#pragma unroll
    for (int w = 0; w < kConsumers; ++w) mf = fmaxf(mf, sm->wm[w][r]);
    const float msafe = mf == -INFINITY ? 0.f : mf;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
#pragma unroll
    for (int w = 0; w < kConsumers; ++w) {
      const float sc = exp2f(sm->wm[w][r] - msafe);
      float4 v = *reinterpret_cast<const float4*>(Om + (w * NT * 8 + r) * kRow + d);
      if (FOLD && (NT == 1 || r >= 8)) {   // the lo terms' part
        const float4 lo = *reinterpret_cast<const float4*>(Om + (w * NT * 8 + r + 4) * kRow + d);
        v.x += lo.x; v.y += lo.y; v.z += lo.z; v.w += lo.w;
      }
      acc.x += v.x * sc; acc.y += v.y * sc; acc.z += v.z * sc; acc.w += v.w * sc;
      l += sm->wl[w][r] * sc;
    }
    if (cl == 1) {
      store(r, d, acc, mf, l);
    } else {
      *reinterpret_cast<float4*>(part + r * D + d) = acc;
      if (d == 0) { part_m[r] = mf; part_l[r] = l; }
    }
  }
  if (cl > 1) {
    cluster_sync();
    // the CTAs share the rows' columns out among themselves
    for (int i = tid * cl + sp; i < GH * (D / 4); i += kDecThreads * cl) {
      const int r = i / (D / 4), d = i % (D / 4) * 4;
      float mj[kMaxCluster];
      float mf = -INFINITY;
#pragma unroll
      for (int j = 0; j < kMaxCluster; ++j) {
        mj[j] = j < cl ? peer_load(peer_smem(part_m + r, j)) : -INFINITY;
        mf = fmaxf(mf, mj[j]);
      }
      const float msafe = mf == -INFINITY ? 0.f : mf;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      float l = 0.f;
#pragma unroll
      for (int j = 0; j < kMaxCluster; ++j) {
        if (j >= cl) break;
        const float sc = exp2f(mj[j] - msafe);
        const float4 v = peer_load4(peer_smem(part + r * D + d, j));
        acc.x += v.x * sc; acc.y += v.y * sc; acc.z += v.z * sc; acc.w += v.w * sc;
        l += peer_load(peer_smem(part_l + r, j)) * sc;
      }
      store(r, d, acc, mf, l);
    }
    cluster_sync();   // the others have read this CTA's part
  }
  leave();
}

// out[row] = sum_p o_p[row] * softmax_p(lse_p[row]); merged lse = logsumexp_p.
template <typename Tin, typename Tout>
__global__ void merge_kernel(const Tin* __restrict__ o_parts, const float* __restrict__ lse_parts,
                             int P, int64_t rows, int d, int64_t pso, int64_t rso, int64_t psl,
                             int64_t rsl, Tout* __restrict__ o, int64_t ors,
                             float* __restrict__ lse, int64_t lrs) {
  const int64_t total = rows * d;
  // Launched as a programmatic dependent of the decode kernel: the blocks may already be
  // resident while that grid drains, and wait here until its partials are visible.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / d;
    const int c = (int)(i - r * d);
    float mx = -INFINITY;
    for (int q = 0; q < P; ++q) mx = fmaxf(mx, lse_parts[q * psl + r * rsl]);
    const float ms = mx == -INFINITY ? 0.f : mx;
    float den = 0.f, acc = 0.f;
    for (int q = 0; q < P; ++q) {
      const float w = __expf(lse_parts[q * psl + r * rsl] - ms);
      den += w;
      if (w != 0.f) acc += w * Elem<Tin>::to_f(o_parts[q * pso + r * rso + c]);
    }
    o[r * ors + c] = Elem<Tout>::from_f(den > 0.f ? acc / den : 0.f);
    if (c == 0 && lse) lse[r * lrs] = den > 0.f ? ms + __logf(den) : -INFINITY;
  }
}

template <typename Tin, typename Tout>
int launch_merge(const void* o_parts, const float* lse_parts, int P, int64_t rows, int d,
                 int64_t pso, int64_t rso, int64_t psl, int64_t rsl, void* o, int64_t ors,
                 float* lse, cudaStream_t s, int64_t lrs = 1) {
  const int64_t total = rows * d;
  if (total == 0) return BSA_OK;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BSA_CHECK_CUDA(cudaLaunchKernelEx(&cfg, merge_kernel<Tin, Tout>, reinterpret_cast<const Tin*>(o_parts),
                                    lse_parts, P, rows, d, pso, rso, psl, rsl,
                                    reinterpret_cast<Tout*>(o), ors, lse, lrs));
  return check_launch("merge_kernel");
}

// Checks that must hold before any arithmetic on the head counts (the split planning divides by
// them): shared by bsa_decode, bsa_decode_static and bsa_decode_workspace_bytes.
int decode_validate_heads(const bsa_decode_params* p, const char* who) {
  BSA_CHECK_ARG(p, "%s: null params", who);
  BSA_CHECK_ARG(p->batch >= 0 && p->hq >= 1 && p->hkv >= 1 && p->hq % p->hkv == 0,
                "%s: bad head counts hq=%d hkv=%d", who, p->hq, p->hkv);
  const int G = p->hq / p->hkv;
  BSA_CHECK_ARG(p->heads_per_cta >= 1 && p->heads_per_cta <= 16 && G % p->heads_per_cta == 0,
                "%s: heads_per_cta=%d must divide the group size %d and be <= 16", who,
                p->heads_per_cta, G);
  BSA_CHECK_ARG(p->d >= 1 && p->max_row_nnz >= 0, "%s: bad sizes d=%d max_row_nnz=%d", who, p->d,
                p->max_row_nnz);
  BSA_CHECK_ARG(p->k_blk_mod >= 0 && (p->k_blk_mod <= 1 || (p->k_blk_rem >= 0 && p->k_blk_rem < p->k_blk_mod)),
                "%s: bad block-cyclic shard %d mod %d", who, p->k_blk_rem, p->k_blk_mod);
  return BSA_OK;
}

// Attended blocks per CTA.  A caller's choice is kept; otherwise a CTA gets as many blocks as
// possible (up to 16: one prologue and one partial per 512 KB of K/V) while the grid still
// fills the machine about twice over (three resident CTAs per SM).
int decode_blocks_per_split(const bsa_decode_params* p) {
  if (p->blocks_per_split > 0) return p->blocks_per_split;
  const int hpc = p->heads_per_cta > 0 ? p->heads_per_cta : 1;
  const long long items = (long long)p->batch * p->hkv * ((p->hq / p->hkv) / hpc);
  const long long want = 2LL * 148 * kMinCtas;
  long long splits = items > 0 ? (want + items - 1) / items : 1;
  if (splits < 1) splits = 1;
  const int nnz = p->max_row_nnz > 0 ? p->max_row_nnz : 1;
  long long bps = (nnz + splits - 1) / splits;
  bps = (bps + 3) / 4 * 4;
  if (bps < 4) bps = 4;
  if (bps > 16) bps = 16;
  return (int)bps;
}

int decode_nsplit(const bsa_decode_params* p) {
  const int bps = decode_blocks_per_split(p);
  const int n = (p->max_row_nnz + bps - 1) / bps;
  return n < 1 ? 1 : n;
}

template <typename T, int D, bool FP8, int NT, bool FOLD>
int launch_decode(const bsa_decode_params* p, int nsplit, int cl, const int32_t* row_start, const int32_t* row_end,
                  cudaStream_t s) {
  Tmap4 tmK, tmV;
  const bool bf16 = p->dtype == BSA_BF16;
  const int eb = FP8 ? 1 : 2;
  using Geo = DecGeo<D, FP8>;
  const uint32_t box_d = FP8 ? D : 64;    // 8-bit tiles are copied in one box, 16-bit ones in 128-byte wide boxes
  int rc = make_tmap_4d(&tmK, p->k, eb, D, p->sk, p->hkv, p->batch, p->k_ss * eb, p->k_sh * eb,
                        p->k_sb * eb, box_d, Geo::kTok, Geo::kSwizzle, bf16);
  if (rc) return rc;
  rc = make_tmap_4d(&tmV, p->v, eb, D, p->sk, p->hkv, p->batch, p->v_ss * eb, p->v_sh * eb,
                    p->v_sb * eb, box_d, Geo::kTok, Geo::kSwizzle, bf16);
  if (rc) return rc;
  bsa_decode_params q = *p;
  q.blocks_per_split = decode_blocks_per_split(p);
  const int max_units = q.blocks_per_split * (p->block_size / Geo::kTok);
  const size_t smem = dec_smem<D, FP8, NT>(max_units);
  auto kern = decode_kernel<T, D, FP8, NT, FOLD>;
  // one value for every call: host threads may launch this kernel with different sizes at the same time
  BSA_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)dec_smem<D, FP8, NT>(kMaxRowBlocks * 64 / Geo::kTok)));
  const int G = p->hq / p->hkv;
  dim3 grid(cl > 1 ? cl : nsplit, p->hkv * (G / p->heads_per_cta), p->batch);
  int* status = wait_status_ptr();
  if (!status) return BSA_E_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (cl > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim = {(unsigned)cl, 1, 1};
    ++cfg.numAttrs;
  }
  if (row_start) {   // behind the prefill kernel of the call
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  BSA_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, tmK, tmV, q, nsplit, cl, max_units, row_start, row_end, status));
  rc = check_launch("decode_kernel");
  if (rc) return rc;
  if (nsplit > 1 && p->o) {
    const int64_t rows = (int64_t)p->batch * p->hq;
    float* ws_lse = p->ws + rows * nsplit * D;
    // partial o: (rows, nsplit, D) -> partition stride D, row stride nsplit*D; rows of o and lse may be
    // strided (e.g. packed side by side in one buffer), batch and head collapse into one row index
    // (decode_run has checked that they do)
    if (bf16)
      return launch_merge<float, __nv_bfloat16>(p->ws, ws_lse, nsplit, rows, D, D, (int64_t)nsplit * D, 1, nsplit,
                                                p->o, p->o_sh, p->lse, s, p->lse_sh);
    return launch_merge<float, __half>(p->ws, ws_lse, nsplit, rows, D, D, (int64_t)nsplit * D, 1, nsplit, p->o,
                                       p->o_sh, p->lse, s, p->lse_sh);
  }
  return BSA_OK;
}

template <typename T>
int launch_decode_t(const bsa_decode_params* p, bool fp8, int nsplit, int cl, const int32_t* row_start,
                    const int32_t* row_end, cudaStream_t s) {
  auto go = [&](auto kernel) { return kernel(p, nsplit, cl, row_start, row_end, s); };
  auto go_heads = [&](auto d, auto kv8) {
    constexpr int D = decltype(d)::value;
    constexpr bool FP8 = decltype(kv8)::value;
    if (p->heads_per_cta > 12) return go(launch_decode<T, D, FP8, 2, false>);
    if (p->heads_per_cta > 8) return go(launch_decode<T, D, FP8, 2, true>);
    if (p->heads_per_cta > 4) return go(launch_decode<T, D, FP8, 1, false>);
    return go(launch_decode<T, D, FP8, 1, true>);
  };
  using D64 = std::integral_constant<int, 64>;
  using D128 = std::integral_constant<int, 128>;
  if (fp8) return p->d == 128 ? go_heads(D128(), std::true_type()) : go_heads(D64(), std::true_type());
  return p->d == 128 ? go_heads(D128(), std::false_type()) : go_heads(D64(), std::false_type());
}

}  // namespace

size_t decode_workspace_bytes(const bsa_decode_params* p) {
  if (decode_validate_heads(p, "bsa_decode_workspace_bytes") != BSA_OK) return 0;
  const int nsplit = decode_nsplit(p);
  if (nsplit <= 1 && p->o) return 0;   // without an output tensor even a single split stays a partial
  return sizeof(float) * (size_t)p->batch * p->hq * nsplit * (p->d + 1);
}

int decode_run(const bsa_decode_params* p, cudaStream_t s) {
  int vrc = decode_validate_heads(p, "bsa_decode");
  if (vrc) return vrc;
  BSA_CHECK_ARG(p->q && p->k && p->v && (p->o || p->ws) && p->crow && p->col, "bsa_decode: null pointer");
  BSA_CHECK_ARG(p->h_pat == 1 || p->h_pat == p->hkv || p->h_pat == p->hq,
                "bsa_decode: pattern has %d heads, expected 1, %d or %d", p->h_pat, p->hkv, p->hq);
  if (p->batch == 0) return BSA_OK;
  if (!(p->dtype == BSA_F16 || p->dtype == BSA_BF16) || !(p->d == 64 || p->d == 128) ||
      !(p->block_size == 64 || p->block_size == 128)) {
    set_error("bsa_decode: needs f16/bf16, head dim 64 or 128 and block size 64 or 128 "
              "(got dtype %d, d %d, block %d)", p->dtype, p->d, p->block_size);
    return BSA_E_UNSUPPORTED;
  }
  const bool fp8 = p->kv_dtype == BSA_F8E4M3;
  BSA_CHECK_ARG(p->kv_dtype == 0 || fp8, "bsa_decode: kv_dtype must be 0 (as q) or BSA_F8E4M3, got %d", p->kv_dtype);
  BSA_CHECK_ARG(!fp8 || (p->k_scale > 0.f && p->v_scale > 0.f), "bsa_decode: e4m3 K/V need positive k_scale and v_scale");
  if (!tma_compatible(p->k, fp8 ? 1 : 2, p->k_ss, p->k_sh, p->k_sb) ||
      !tma_compatible(p->v, fp8 ? 1 : 2, p->v_ss, p->v_sh, p->v_sb)) {
    set_error("bsa_decode: K/V need a 16-byte aligned base and strides that are multiples of 16 bytes");
    return BSA_E_UNSUPPORTED;
  }
  const int bps = decode_blocks_per_split(p);
  if (bps * p->block_size > kMaxTokens) {
    set_error("bsa_decode: blocks_per_split=%d too large (limit %d tokens per CTA)", bps, kMaxTokens);
    return BSA_E_TOOBIG;
  }
  const int nsplit = decode_nsplit(p);
  BSA_CHECK_ARG((nsplit == 1 && p->o) || p->ws, "bsa_decode: workspace required for %d splits", nsplit);
  if (nsplit > 1 && p->o &&
      (p->o_sb != (int64_t)p->hq * p->o_sh || (p->lse && p->lse_sb != (int64_t)p->hq * p->lse_sh))) {
    set_error("bsa_decode: with several splits o and lse need batch stride = heads x head stride");
    return BSA_E_UNSUPPORTED;
  }
  // Where the whole grid is resident at once with some room to spare, up to eight splits are a cluster whose
  // CTAs merge their parts over distributed shared memory: no partials and no second launch.  In a larger
  // grid waiting for a cluster's worth of room costs more than the second launch.  (Sequences of 3000 to 4096
  // tokens, 32/8 heads, D 128, 64 CTAs each: 1: 13.3 -> 11.3 us, 2: 13.3 -> 11.9, 4: 14.0 -> 13.3, 6: 15.4 ->
  // 13.3, 8: 17.1 -> 21.5 us; 64 of 1024 to 8192 tokens: 69 -> 71 us.  Those are eight splits; two to seven,
  // one sequence and as many as the limit takes: 2: 8.5 -> 7.8, 24: 12.2 -> 10.0; 4: 9.4 -> 8.2, 12: 12.8 -> 10.5;
  // 7: 10.3 -> 8.7, 6: 12.8 -> 11.0 us; e4m3 the same.)
  const long long ctas = (long long)p->batch * (p->hq / p->heads_per_cta) * nsplit;
  const int resident = fp8 && p->d == 128 && p->heads_per_cta > 8 ? 2 : kMinCtas;   // the kernel's launch bounds
  const int cl = p->o && nsplit > 1 && nsplit <= kMaxCluster && ctas <= kClusterCtas * resident ? nsplit : 1;
  if (p->dtype == BSA_BF16) return launch_decode_t<__nv_bfloat16>(p, fp8, cl > 1 ? 1 : nsplit, cl, nullptr, nullptr, s);
  return launch_decode_t<__half>(p, fp8, cl > 1 ? 1 : nsplit, cl, nullptr, nullptr, s);
}

// The sequences of a packed batch that have one query token.  A CTA walks a whole pattern row (there
// is no scratch for partials); its list holds every block of the pattern's longest possible row, which is
// kMaxRowBlocks at most (sm100_fwd_supported: rows or keys of the call are bounded by it).  (Two or four CTAs
// per row as a cluster: 163 and 221 us for the batch of sm100_fwd's comment, against 135 at the time.)
int decode_packed_rows(const bsa_fwd_params* f, cudaStream_t s) {
  bsa_decode_params p = {};
  p.q = f->q; p.k = f->k; p.v = f->v; p.o = f->o; p.lse = f->lse;
  p.q_sb = f->q_ss; p.q_sh = f->q_sh;
  p.k_sb = f->k_sb; p.k_ss = f->k_ss; p.k_sh = f->k_sh;
  p.v_sb = f->v_sb; p.v_ss = f->v_ss; p.v_sh = f->v_sh;
  p.o_sb = f->o_ss; p.o_sh = f->o_sh;
  p.lse_sb = 1; p.lse_sh = f->lse_sh;
  p.batch = f->batch; p.hq = f->hq; p.hkv = f->hkv; p.d = f->d; p.sk = f->sk;
  p.k_start = f->k_start; p.k_end = f->k_end;
  p.crow = f->crow; p.col = f->col; p.crow_sh = f->crow_sh; p.col_sh = f->col_sh;
  p.h_pat = f->h_pat; p.n_rows = f->n_rows; p.block_size = f->block_size;
  // the heads of a CTA share a block list
  const int G = f->hq / f->hkv;
  p.heads_per_cta = 1;
  if (f->h_pat != f->hq)
    for (int c = 2; c <= G && c <= 16; ++c)
      if (G % c == 0) p.heads_per_cta = c;
  // columns ascend and a causal row sees no block past the sequence: its first cdiv(sk, 64) entries do
  p.max_row_nnz = f->n_rows < cdiv_i(f->sk, 64) ? f->n_rows : cdiv_i(f->sk, 64);
  p.blocks_per_split = p.max_row_nnz;
  p.dtype = f->dtype;
  p.sm_scale = f->sm_scale;
  if (p.dtype == BSA_BF16) return launch_decode_t<__nv_bfloat16>(&p, false, 1, 1, f->q_start, f->q_end, s);
  return launch_decode_t<__half>(&p, false, 1, 1, f->q_start, f->q_end, s);
}

int merge_partials(const void* o_parts, const float* lse_parts, int P, int64_t rows, int d,
                   int64_t pso, int64_t rso, int64_t psl, int64_t rsl, void* o, int64_t ors,
                   float* lse, int dtype, cudaStream_t s) {
  BSA_CHECK_ARG(o_parts && lse_parts && o, "bsa_merge_partials: null pointer");
  BSA_CHECK_ARG(P >= 1 && rows >= 0 && d >= 1, "bsa_merge_partials: bad sizes P=%d d=%d", P, d);
  switch (dtype) {
    case BSA_F16: return launch_merge<__half, __half>(o_parts, lse_parts, P, rows, d, pso, rso, psl, rsl, o, ors, lse, s);
    case BSA_BF16: return launch_merge<__nv_bfloat16, __nv_bfloat16>(o_parts, lse_parts, P, rows, d, pso, rso, psl, rsl, o, ors, lse, s);
    case BSA_F32: return launch_merge<float, float>(o_parts, lse_parts, P, rows, d, pso, rso, psl, rsl, o, ors, lse, s);
  }
  set_error("bsa_merge_partials: unknown dtype %d", dtype);
  return BSA_E_BADARG;
}

}  // namespace bsa

namespace bsa {
// Device address of the status word of the current device (the symbol name is
// only a host-side handle; kernels get the real address as an argument).
int* wait_status_ptr() {
  static int* cache[64] = {nullptr};
  static std::mutex mu;   // entry points may be called from several host threads
  std::lock_guard<std::mutex> lock(mu);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    set_error("cudaGetDevice failed or device index out of range");
    return nullptr;
  }
  if (!cache[dev]) {
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_wait_status);
    if (e != cudaSuccess) {
      set_error("cudaGetSymbolAddress(g_wait_status) failed: %s", cudaGetErrorString(e));
      return nullptr;
    }
    cache[dev] = static_cast<int*>(ptr);
  }
  return cache[dev];
}

static int* g_mirror_host[64] = {nullptr};   // the registered mirror word of each device

int read_wait_status(int* out, int reset) {
  BSA_CHECK_ARG(out, "bsa_wait_status: null pointer");
  BSA_CHECK_CUDA(cudaDeviceSynchronize());
  BSA_CHECK_CUDA(cudaMemcpyFromSymbol(out, g_wait_status, sizeof(int)));
  if (reset && *out != 0) {
    const int zero = 0;
    BSA_CHECK_CUDA(cudaMemcpyToSymbol(g_wait_status, &zero, sizeof(int)));
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && g_mirror_host[dev])
      *reinterpret_cast<volatile int*>(g_mirror_host[dev]) = 0;
  }
  return BSA_OK;
}

int set_wait_status_mirror(int* host_word) {
  int dev = 0;
  BSA_CHECK_CUDA(cudaGetDevice(&dev));
  BSA_CHECK_ARG(dev >= 0 && dev < 64, "bsa_set_wait_status_mirror: device index out of range");
  int* dptr = nullptr;
  if (host_word) {
    cudaError_t e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&dptr), host_word, 0);
    if (e != cudaSuccess || !dptr) {
      (void)cudaGetLastError();
      set_error("bsa_set_wait_status_mirror: the word must be page-locked host memory that the device "
                "can address (%s)", cudaGetErrorString(e));
      return BSA_E_BADARG;
    }
  }
  BSA_CHECK_CUDA(cudaMemcpyToSymbol(g_wait_status, &dptr, sizeof(dptr), 2 * sizeof(int)));
  g_mirror_host[dev] = host_word;
  return BSA_OK;
}

// A wait that nothing will ever satisfy, with a short limit: exercises the give-up path
// (status block, mirror word, no-op behaviour of later launches) without faulting the GPU.
__global__ void wait_timeout_selftest_kernel(int* status, uint64_t limit_ns) {
  __shared__ uint64_t bar;
  if (*reinterpret_cast<volatile int*>(status) != 0) return;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
    mbar_wait(&bar, 0, status, 900, limit_ns);   // nobody arrives
  }
}

int selftest_wait_timeout(uint32_t limit_us, cudaStream_t s) {
  BSA_CHECK_ARG(limit_us >= 1 && limit_us <= 100000, "bsa_selftest_wait_timeout: limit must be 1..100000 us");
  int* status = wait_status_ptr();
  if (!status) return BSA_E_CUDA;
  wait_timeout_selftest_kernel<<<1, 32, 0, s>>>(status, (uint64_t)limit_us * 1000ull);
  return check_launch("wait_timeout_selftest_kernel");
}
}  // namespace bsa

// ---------------------------------------------------------------------------
// Decode without any allocation by the caller.
//
// Some hosts of this library cannot hand it scratch memory: a serving runtime
// that has pinned its whole device-memory budget to the KV cache, a plugin
// loaded into a process whose allocator it must not touch, a language binding
// that only passes through the tensors it was given.  For them the split-KV
// partials live in a fixed array that is part of the library image.  Every GPU
// that loads the library carries the array (kStaticScratchBytes) until the
// process exits.
// ---------------------------------------------------------------------------
namespace bsa {

constexpr size_t kStaticScratchBytes = size_t(8) << 20;  // 8 MiB
static __device__ __align__(256) float g_decode_scratch[kStaticScratchBytes / sizeof(float)];

// Device address of g_decode_scratch on the current device.  In host code the
// array's name is only a handle for the runtime, not an address a kernel can
// use, so the address is looked up once per device (with that device current)
// and handed to the kernels as an ordinary pointer.
static float* static_scratch_ptr() {
  static float* cache[64] = {nullptr};
  static std::mutex mu;   // entry points may be called from several host threads
  std::lock_guard<std::mutex> lock(mu);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    set_error("bsa_decode_static: cudaGetDevice failed or device index out of range");
    return nullptr;
  }
  if (!cache[dev]) {
    float* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&ptr, g_decode_scratch);
    if (e != cudaSuccess || ptr == nullptr) {
      set_error("bsa_decode_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return nullptr;
    }
    cache[dev] = ptr;
  }
  return cache[dev];
}

size_t decode_static_capacity() { return kStaticScratchBytes; }

int decode_run_static(const bsa_decode_params* p, cudaStream_t s) {
  int vrc = decode_validate_heads(p, "bsa_decode_static");
  if (vrc) return vrc;
  const size_t need = decode_workspace_bytes(p);
  if (need > kStaticScratchBytes) {
    set_error("bsa_decode_static: this call needs %zu bytes of split-KV scratch but the built-in "
              "array holds %zu; lower batch*heads, raise blocks_per_split, or use bsa_decode with a "
              "caller-provided workspace", need, (size_t)kStaticScratchBytes);
    return BSA_E_TOOBIG;
  }
  float* scratch = static_scratch_ptr();
  if (!scratch) return BSA_E_CUDA;
  bsa_decode_params q = *p;
  q.ws = scratch;  // every (sequence, head, split) slot in use is rewritten by the kernel
  return decode_run(&q, s);
}

}  // namespace bsa
