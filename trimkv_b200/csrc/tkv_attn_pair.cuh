// The core of the query-resident attention kernels on tcgen05 + TMEM: two tiles of 128 query rows per CTA (two blocks of rows,
// or two maps of the same rows) against tiles of 128 keys, an online softmax in between.
//
//   S_t[128 x 128] = Q_t . K(j)^T      A = Q (shared memory, staged once), B = K as TMA wrote it; TMEM columns 128 t
//   softmax        warpgroup t, thread = row: the row of S is read once into registers, P in the 16-bit type is written over
//                  the first half of S's columns, so no value of a row ever crosses threads or goes through shared memory
//   O_t           += P_t . V(j)        A = P from TMEM, B = V read MN-major from the bytes TMA wrote; columns 256 + 128 t
// What bounds it is the exponential unit (16 results per SM and cycle: 1024 cycles for a tile, the same as its two products
// of 128 dims) and, in a chain product - softmax - product, the length of the chain: two independent chains share the units.
// One tile with two threads per row, S of the next key tile computed ahead and P through shared memory took 3800 cycles a tile:
// every step crossed four barriers of 256 arrivals and waited for P . V of the step before; in two tiles it takes 2500.  512 queries of
// 8 x 16 heads against 4608 keys 233 -> 187 us; differential with its preparation, 8192 tokens, 16 heads, window 4096, 652 -> 464 us;
// two-part, 2 x 4096 tokens, 32 heads, 591 -> 441 us.  With products issued by an elected lane of a whole warp (17 to 21 cycles each
// instead of 51 in a branch of one lane) 187 -> 166 us, and a differential and a latent layer of the last two 635 -> 606 and 1012 -> 989 us with
// their library products.  The power of the chip bounds it now: 4150 -> 3240 cycles for a block of keys
// by fewer arrivals brought the SM clock from 1.80 to 1.62 GHz and the same 166 us.  Sums are taken in the order of those kernels: the
// results are the same bit for bit.
//
// P . V of a step reads the TMEM columns that S of the next one writes.  PTX promises an order of two products only where they have
// one accumulator and shape, so S is issued when P . V is complete; behind S of a step O may therefore be rescaled.  O is rescaled
// only when a row's maximum grew by more than 2^8 since its reference was fixed, which is rare after the first tiles.
//
// Roles: warps 0-3 and 4-7 softmax of tiles 0 and 1; warp 8 issues the products, warp 9 the copies (one lane each).  Every wait
// is bounded.
#pragma once
#include "tkv_attn_block.cuh"
#include "tkv_common.cuh"

namespace tkv {

constexpr int kPairThreads = kDaSoftmaxThreads + 64;

struct PairSmem {
  uint64_t full_k[3], empty_k[3], full_v[2], empty_v[2], s_ready[2], p_half[2], p_ready[2], o_ready[2], meet;
  uint32_t tmem_base;
  int abort_flag;
  float red[2][kDaTile];
};

// KH, VH: 64-element pieces of a key and of a value.  kTwoKeys: every tile has keys of its own (the maps of differential
// attention), side by side in a stage.  As many stages as fit, two of K before two of V before three of K.
template <int KH_, int VH_, bool kTwoKeys_> struct PairShape {
  static constexpr int KH = KH_, VH = VH_;
  static constexpr bool kTwoKeys = kTwoKeys_;
  static constexpr int kTileQ = KH * kDaHalf, kTileK = KH * kDaHalf, kStageK = kTileK * (kTwoKeys ? 2 : 1), kStageV = VH * kDaHalf;
  static constexpr int kMost = 232448 - (int)sizeof(PairSmem);
  static constexpr int kNV = 2 * (kTileQ + kStageK + kStageV) <= kMost ? 2 : 1;
  static constexpr int kNK = 2 * kTileQ + 3 * kStageK + kNV * kStageV <= kMost ? 3 : 2;
  static constexpr int kBytes = 2 * kTileQ + kNK * kStageK + kNV * kStageV + (int)sizeof(PairSmem);
  static_assert(kBytes <= 232448, "shared memory of the kernel");
  static __device__ __forceinline__ uint8_t* q(uint8_t* base, int t) { return base + t * kTileQ; }
  static __device__ __forceinline__ uint8_t* k(uint8_t* base, int j) { return base + 2 * kTileQ + (j % kNK) * kStageK; }
  static __device__ __forceinline__ uint8_t* v(uint8_t* base, int j) { return base + 2 * kTileQ + kNK * kStageK + (j % kNV) * kStageV; }
  static __device__ __forceinline__ PairSmem* smem(uint8_t* base) {
    return reinterpret_cast<PairSmem*>(base + 2 * kTileQ + kNK * kStageK + kNV * kStageV);
  }
};

// Key tiles [j0, j1) of a tile of rows, counted from the CTA's first one; empty: no products, and O is not written.
struct PairRange { int j0, j1; };

// Two fp32 operations in one instruction.
__device__ __forceinline__ float2 pair_fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tfma.rn.f32x2 r, a, b, c;\n\t"
      "mov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
template <bool kBf16> __device__ __forceinline__ uint32_t pair_pack2(float a, float b) {
  if (kBf16) return da_pack2(a, b);
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <bool kBf16> __device__ __forceinline__ uint32_t pair_idesc(int n, int b_mn_major) {   // A, B of one 16-bit type, fp32 D, M = 128
  return (1u << 4) | ((kBf16 ? 1u : 0u) << 7) | ((kBf16 ? 1u : 0u) << 10) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(n >> 3) << 17) |
         ((128u >> 4) << 24);
}

__device__ __forceinline__ void pair_init(PairSmem* sm) {
  for (int i = 0; i < 3; ++i) { mbar_init(&sm->full_k[i], 1); mbar_init(&sm->empty_k[i], 1); }
  for (int i = 0; i < 2; ++i) {
    mbar_init(&sm->full_v[i], 1); mbar_init(&sm->empty_v[i], 1);
    mbar_init(&sm->s_ready[i], 1); mbar_init(&sm->o_ready[i], 1);
    mbar_init(&sm->p_half[i], 4); mbar_init(&sm->p_ready[i], 4);   // one arrival per warp of the tile
  }
  mbar_init(&sm->meet, kDaSoftmaxThreads / 32);
  sm->abort_flag = 0;
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Copies of nt key tiles; load_k(j) and load_v(j) start those of a tile.  *nk, *nv: tiles started.
template <typename Shape, typename LoadK, typename LoadV>
__device__ __forceinline__ bool pair_copies(PairSmem* sm, int nt, LoadK load_k, LoadV load_v, int* nk, int* nv) {
  volatile int* abort_flag = &sm->abort_flag;
  for (int i = 0; i <= nt; ++i) {                          // K one tile ahead of V
    if (i < nt) {
      if (!mbar_wait_or_abort(&sm->empty_k[i % Shape::kNK], ((i / Shape::kNK) & 1) ^ 1, abort_flag)) return false;
      mbar_expect_tx(&sm->full_k[i % Shape::kNK], Shape::kStageK);
      load_k(i);
      ++*nk;
    }
    if (i > 0) {
      const int j = i - 1;
      if (!mbar_wait_or_abort(&sm->empty_v[j % Shape::kNV], ((j / Shape::kNV) & 1) ^ 1, abort_flag)) return false;
      mbar_expect_tx(&sm->full_v[j % Shape::kNV], Shape::kStageV);
      load_v(j);
      ++*nv;
    }
  }
  return true;
}

// The products, in the order  P.V of tile 0 - S of tile 0 for the next keys - P.V of tile 1 - S of tile 1 for the next keys.  S waits
// until the P.V before it is complete, since it is written over the weights which that reads.  That costs the two kernels with keys of
// 128 dims 3 % (a warp of its own for each tile's products: 25 %, as its polling takes issue slots from the softmax; S in two halves,
// the one beside the weights first: 20 %, as products of 64 columns take as long as of 128).  Stages are given back where a copy will
// wait for them, a single stage of V before S of tile 1: its copy is then ready in time (two-part 490 -> 441 us).
// Run by a whole warp.
template <typename Shape, bool kBf16>
__device__ __forceinline__ bool pair_products(PairSmem* sm, uint8_t* base, uint32_t tmem_, int nt_, const PairRange* range_) {
  volatile int* abort_flag = &sm->abort_flag;
  const uint32_t idesc_s = pair_idesc<kBf16>(128, 0), idesc_pv = pair_idesc<kBf16>(Shape::VH * 64, 1);
  const uint32_t tmem = warp_uniform(tmem_);
  const int nt = warp_uniform(nt_);
  const PairRange range[2] = {{warp_uniform(range_[0].j0), warp_uniform(range_[0].j1)}, {warp_uniform(range_[1].j0), warp_uniform(range_[1].j1)}};
  const uint64_t q_desc = make_desc(smem_u32(Shape::q(base, 0)), 16, 1024, 2), k_desc = make_desc(smem_u32(Shape::k(base, 0)), 16, 1024, 2),
                 v_desc = make_desc(smem_u32(Shape::v(base, 0)), kDaHalf, 1024, 2);   // in units of 16 bytes
  auto weighted = [&](int t, int j, int k0, int k1) {      // 16 keys per product: 8 columns of P, 2048 bytes down the V tile
    const uint64_t v = v_desc + (uint32_t)(j % Shape::kNV) * (Shape::kStageV >> 4);
#pragma unroll
    for (int k = k0; k < k1; ++k) umma_ts(tmem + 256 + 128 * t, tmem + 128 * t + 8 * k, v + k * 128, idesc_pv, (j > range[t].j0 || k > 0));
  };
  auto scores = [&](int t, int j) {                        // 16 dims per product
    const uint64_t q = q_desc + t * (Shape::kTileQ >> 4);
    const uint64_t k_ = k_desc + (uint32_t)(j % Shape::kNK) * (Shape::kStageK >> 4) + (Shape::kTwoKeys ? t * (Shape::kTileK >> 4) : 0);
#pragma unroll
    for (int k = 0; k < Shape::KH * 4; ++k) {
      const uint32_t off = (k >> 2) * (kDaHalf >> 4) + (k & 3) * 2;
      umma(tmem + 128 * t, q + off, k_ + off, idesc_s, k > 0);
    }
  };
  auto wait_for = [&](uint64_t* bar, int t, int j) {
    if (!warp_wait(bar, (j - range[t].j0) & 1, abort_flag)) return false;
    tc_fence_after();
    return true;
  };
  auto in = [&](int t, int j) { return j >= range[t].j0 && j < range[t].j1; };
  for (int j = -1; j < nt; ++j) {
    const int jn = j + 1;
    if (j >= 0 && !warp_wait(&sm->full_v[j % Shape::kNV], (j / Shape::kNV) & 1, abort_flag)) return false;
    if (jn < nt && !warp_wait(&sm->full_k[jn % Shape::kNK], (jn / Shape::kNK) & 1, abort_flag)) return false;
    tc_fence_after();
    const bool give_v = j >= 0 && j + Shape::kNV < nt;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (in(t, j)) {
        if (!wait_for(&sm->p_half[t], t, j)) return false; // the first half of P runs under the exponentials of the second
        if (elect_one()) weighted(t, j, 0, 4);
        __syncwarp();
        if (!wait_for(&sm->p_ready[t], t, j)) return false;
        if (elect_one()) {
          weighted(t, j, 4, 8);
          umma_commit(&sm->o_ready[t]);
        }
        __syncwarp();
      }
      if (Shape::kNV == 1 && t == 1 && give_v) {
        if (elect_one()) umma_commit(&sm->empty_v[0]);
        __syncwarp();
      }
      if (in(t, jn)) {
        if (in(t, j) && !wait_for(&sm->o_ready[t], t, j)) return false;
        tc_fence_after();
        if (elect_one()) {
          scores(t, jn);
          umma_commit(&sm->s_ready[t]);
        }
        __syncwarp();
      }
    }
    if (elect_one()) {
      if (Shape::kNV > 1 && give_v) umma_commit(&sm->empty_v[j % Shape::kNV]);
      if (jn + Shape::kNK < nt) umma_commit(&sm->empty_k[jn % Shape::kNK]);
    }
    __syncwarp();
  }
  return true;
}

// Softmax of tile t: this thread's row sees columns [lo, hi) of the keys, whose column col0 is the first of key tile 0; columns
// from len on belong to nobody.  Leaves the row's sum of weights, O in TMEM.  kZeroEmpty: a row whose scores are all -inf has
// weights 0 (else NaN, as the quotient of zeros).  False if a wait ran out.
template <typename Shape, bool kBf16, bool kZeroEmpty>
__device__ __forceinline__ bool pair_softmax(PairSmem* sm, uint8_t* base, uint32_t tmem, int t, PairRange range, int lo, int hi, int col0,
                                             int len, float scale_log2, float* sum) {
  volatile int* abort_flag = &sm->abort_flag;
  const int row = threadIdx.x & (kDaTile - 1), lane = threadIdx.x & 31;
  const uint32_t lane_base = tmem + ((uint32_t)(row & ~31) << 16);
  const uint32_t s_addr = lane_base + 128 * t, o_addr = lane_base + 256 + 128 * t;
  float m_ref = -INFINITY, l_sum[2] = {0.f, 0.f};          // reference maximum (log2 domain); weights of each half of the columns
  for (int j = range.j0; j < range.j1; ++j) {
    bool ok = mbar_wait_or_abort(&sm->s_ready[t], (j - range.j0) & 1, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) return false;
    tc_fence_after();
    const int t0 = col0 + j * kDaTile, first = lo - t0, end = hi - t0;
    uint32_t sv[128];
#pragma unroll
    for (int c = 0; c < 4; ++c) da_ld32_nowait(s_addr + 32 * c, sv + 32 * c);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    bool blank = false;                                    // no column of the tile visible
    if (first > 0 || end < kDaTile) {
      blank = end <= max(first, 0) || first >= kDaTile;
#pragma unroll
      for (int i = 0; i < 128; ++i)
        if (i < first || i >= end) sv[i] = 0xff800000u;
    }
    float mr[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < 128; i += 8)
#pragma unroll
      for (int e = 0; e < 4; ++e) mr[e] = fmaxf(fmaxf(mr[e], __uint_as_float(sv[i + 2 * e])), __uint_as_float(sv[i + 2 * e + 1]));
    const float m_tile = fmaxf(fmaxf(mr[0], mr[1]), fmaxf(mr[2], mr[3])) * scale_log2;   // the scale is positive (checked on the host)
    const bool grow = m_tile > m_ref + kDaRescaleGap || (m_ref == -INFINITY && m_tile > -INFINITY);
    if (__any_sync(0xffffffffu, grow)) {
      const float m_new = fmaxf(m_ref, m_tile);
      if (j > range.j0) {
        const float alpha = (m_ref == -INFINITY) ? 1.0f : exp2_weight(m_ref - m_new);    // O of such a row is still zero
#pragma unroll 1
        for (int c = 0; c < 4 * Shape::VH; ++c) {          // few at a time: the scores are held in registers meanwhile
          float o[16];
          tmem_ld16(o_addr + 16 * c, o);
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] *= alpha;
          tmem_st16_nowait(o_addr + 16 * c, o);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        l_sum[0] *= alpha; l_sum[1] *= alpha;
      }
      m_ref = m_new;
    }
    const float neg_m = (m_ref == -INFINITY && (kZeroEmpty || blank)) ? 0.f : -m_ref;
    // Rows of the last V tile beyond len may hold anything (stale rows, another request's): their weight is zero, but 0 x NaN
    // would poison the product, so they are cleared.
    if (t0 + kDaTile > len) {
      ok = mbar_wait_or_abort(&sm->full_v[j % Shape::kNV], (j / Shape::kNV) & 1, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) return false;
      if (t0 + row >= len) {
        uint8_t* vt = Shape::v(base, j) + row * 128;
#pragma unroll
        for (int h = 0; h < Shape::VH; ++h)
#pragma unroll
          for (int c = 0; c < 8; ++c) st16(vt + h * kDaHalf + c * 16, make_uint4(0, 0, 0, 0));
      }
      fence_async_smem();
    }
    const float2 scale2 = make_float2(scale_log2, scale_log2), neg2 = make_float2(neg_m, neg_m);
    float ls[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c % 2 == 0) ls[0] = ls[1] = ls[2] = ls[3] = 0.f;
      float w[16];                                         // pairs of 16-bit weights
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float2 z = pair_fma2(make_float2(__uint_as_float(sv[c * 32 + i]), __uint_as_float(sv[c * 32 + i + 1])), scale2, neg2);
        const float x = exp2_weight(z.x), y = exp2_weight(z.y);
        ls[(i >> 1) & 3] += x + y;
        w[i >> 1] = __uint_as_float(pair_pack2<kBf16>(x, y));
      }
      tmem_st16_nowait(s_addr + 16 * c, w);
      if (c % 2 == 1) {                                    // half of P is there
        l_sum[c >> 1] += (ls[0] + ls[1]) + (ls[2] + ls[3]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) da_arrive(c == 1 ? &sm->p_half[t] : &sm->p_ready[t]);
      }
    }
  }
  if (range.j1 > range.j0) {
    const bool ok = mbar_wait_or_abort(&sm->o_ready[t], (range.j1 - 1 - range.j0) & 1, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) return false;
    tc_fence_after();
  }
  *sum = l_sum[0] + l_sum[1];
  return true;
}

// Whole warps of both warpgroups wait for one another; false if the wait ran out.
__device__ __forceinline__ bool pair_meet(PairSmem* sm, int phase) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) da_arrive(&sm->meet);
  const bool ok = mbar_wait_or_abort(&sm->meet, phase & 1, &sm->abort_flag);
  return (bool)__all_sync(0xffffffffu, ok);
}

// Whether CTAs of two tiles of rows take less time than CTAs of one: a CTA per SM at a time, 2.6 us per key tile for a pair against
// 1.64 us for a tile with the chain of its own when measured (64 segments of 192 rows, 33 key tiles: 96 us as 64 pairs, 62 us as 128
// tiles; 64 segments of 2048 rows: 373 us as 512 pairs, 430 us as 1024 tiles).  Products issued by an elected lane made both shorter, 60 us
// as those 128 tiles and 332 us as those 512 pairs, and the line was left where it is.  Two-part keys of 192 dims: 3.7 and 2.6 us (2 x 4096 tokens, 32
// heads: 441 and 591 us; 1500 tokens, 16 heads: 48 and 52 us); of 128 dims the ratio is lower, and 6000 tokens of 8 heads, 192 pairs or
// 376 tiles, would take 118 us instead of 148.  CTAs count as equally long, which those of a prompt without a past are not: 16 segments of
// 1536 rows take 41 us as 96 pairs, 37 us as 192 tiles.  One tile only is never a pair.
inline bool pair_is_faster(int64_t tiles, int64_t pairs) { return pairs < tiles && (pairs + 147) / 148 * 8 < (tiles + 147) / 148 * 5; }

// TMEM is given back; an aborting CTA first waits for the copies it started.
template <typename Shape>
__device__ __forceinline__ void pair_finish(PairSmem* sm, uint32_t tmem, int nk, int nv) {
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == kDaSoftmaxThreads + 32 && *(volatile int*)&sm->abort_flag != 0) {
    for (int i = max(0, nk - Shape::kNK); i < nk; ++i) mbar_wait(&sm->full_k[i % Shape::kNK], (i / Shape::kNK) & 1);
    for (int i = max(0, nv - Shape::kNV); i < nv; ++i) mbar_wait(&sm->full_v[i % Shape::kNV], (i / Shape::kNV) & 1);
  }
  __syncthreads();
  if ((threadIdx.x >> 5) == 8)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kDaTmemCols));
}

}  // namespace tkv
