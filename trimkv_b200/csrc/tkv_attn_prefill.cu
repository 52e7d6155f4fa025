// Query-resident varlen GQA attention for many query tokens per request (prompt passes, pieces of a chunked
// prefill) on tcgen05 + TMEM, K/V streamed once per query block by TMA with an online softmax.
//
// What flash_attn_varlen_func(causal=True) computes for the reference when Q > 1
// (src/trimkv/attn/flash_attn.py:118-145): segment s = (request, KV head) holds seg_len[s] cached tokens including the
// q_tokens new ones; query row R = token * G + head of the segment sees its first seg_len - q_tokens + token + 1
// tokens (bottom-right aligned causal mask).
//
// One CTA = (segment, block of 256 query rows) as two tiles of 128 rows on the core of tkv_attn_pair.cuh.  A tile's key range
// ends with the last key its rows may see.  No workspace, no merge kernel.  Every mbarrier wait is bounded; on expiry the CTA
// records TKV_DEV_TIMEOUT, drains its copies, frees its TMEM and returns.
#include <cuda.h>
#include "tkv_attn.cuh"
#include "tkv_attn_pair.cuh"

namespace tkv {

constexpr int kPfTile = 128;                  // query rows per tile, cached tokens per tile
constexpr int kPfRows = 2 * kPfTile;          // query rows per CTA
using PfShape = PairShape<2, 2, false>;

// grid.x = nseg * nblocks, segment-major: the query blocks of one segment are neighbours in launch order, so they run
// at the same time and the K/V tiles they all stream are fetched from HBM once and then found in L2 (with the blocks of
// different segments side by side instead, a long causal pass re-read its K/V from HBM once per block and was bound
// by that).  Within a segment the blocks go in descending order: the last block of a causal pass sees the most tokens,
// so the longest CTAs start first.
template <int kDtype>
__global__ void __launch_bounds__(kPairThreads, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, AttnParams p,
                    int nseg, int nblocks) {
  extern __shared__ __align__(1024) uint8_t base[];
  constexpr bool kBf16 = kDtype == TKV_BF16;
  grid_dependency_wait();
  grid_launch_dependents();
  const int seg = (int)(blockIdx.x / (unsigned)nblocks);
  const int blk = nblocks - 1 - (int)(blockIdx.x % (unsigned)nblocks);
  const int tid = threadIdx.x, warp = tid >> 5;
  const bool is_row = warp < 8;
  const int t = (tid >> 7) & 1, row = tid & (kPfTile - 1);
  const int G = p.hq / p.hkv;
  const int b = seg / p.hkv, h = seg - b * p.hkv;
  int len = p.seg_len != nullptr ? p.seg_len[seg] : p.max_len;
  if (p.seg_len != nullptr && len > p.max_len) {
    if (tid == 0 && blk == 0) report(p.status, TKV_DEV_LEN_BOUND);
    len = p.max_len;
  }
  if ((smem_u32(base) & 1023u) != 0) {                     // the swizzled tiles need it; the launch gives it
    if (tid == 0) report(p.status, TKV_DEV_TIMEOUT);
    return;
  }
  const int R = blk * kPfRows + t * kPfTile + row;         // this thread's query row of the segment
  const bool row_valid = is_row && R < p.rows;
  const int token = row_valid ? R / G : 0, head = h * G + (row_valid ? R - token * G : 0);
  // cached tokens this row may see, and the key tiles that any row of a tile may see (CTA-uniform)
  const int vis = row_valid ? max(0, min(len, len - p.q_tokens + token + 1)) : 0;
  PairRange range[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int first = blk * kPfRows + i * kPfTile, last = min(first + kPfTile, p.rows) - 1;
    const int most = first < p.rows ? max(0, min(len, len - p.q_tokens + last / G + 1)) : 0;
    range[i] = {0, (most + kPfTile - 1) / kPfTile};
  }
  const int ntiles = max(range[0].j1, range[1].j1);
  char* const out_row = p.out + (((int64_t)b * p.q_tokens + token) * p.hq + head) * 256;
  if (ntiles == 0) {                                       // nothing visible (an empty segment): zeros
    if (row_valid)
      for (int c = 0; c < 16; ++c) st16(out_row + c * 16, make_uint4(0, 0, 0, 0));
    return;
  }

  PairSmem* sm = PfShape::smem(base);
  const int64_t row0 = (int64_t)seg * p.cap;
  if (tid == 0) pair_init(sm);
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)), "r"(kDaTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  } else if (is_row && range[t].j1 > 0) {
    // Q rows as the A operand: K-major with 128-byte swizzle (the layout TMA gives the K tiles)
    const char* qp = p.q + ((int64_t)b * p.q_sb + (int64_t)token * p.q_st + (int64_t)head * p.q_sh) * 2;
    uint8_t* q_s = PfShape::q(base, t);
#pragma unroll
    for (int c = 0; c < 16; ++c) st16(q_s + da_swz(row, c), row_valid ? ld16(qp + c * 16) : make_uint4(0, 0, 0, 0));
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;

  int k_issued = 0, v_issued = 0;                          // copying lane: tiles whose copies have been started
  bool ok = true;
  if (warp == 8) {
    if ((tid & 31) == 0) ok = pair_products<PfShape, kBf16>(sm, base, tmem, ntiles, range);
    __syncwarp();
  } else if (warp == 9) {
    if ((tid & 31) == 0) {
      auto load = [&](uint8_t* to, const CUtensorMap* map, uint64_t* bar, int j) {
        tma_load_2d(to, map, bar, 0, (int)(row0 + j * kPfTile));
        tma_load_2d(to + kDaHalf, map, bar, 64, (int)(row0 + j * kPfTile));
      };
      ok = pair_copies<PfShape>(sm, ntiles, [&](int j) { load(PfShape::k(base, j), &map_k, &sm->full_k[j % PfShape::kNK], j); },
                                [&](int j) { load(PfShape::v(base, j), &map_v, &sm->full_v[j % PfShape::kNV], j); }, &k_issued, &v_issued);
    }
    __syncwarp();
  } else {
    float sum = 0.f;
    ok = pair_softmax<PfShape, kBf16, false>(sm, base, tmem, t, range[t], 0, vis, 0, len, p.scale_log2, &sum);
    if (ok) {                                              // O / sum -> out; a tile that sees nothing is zeros
      const float inv = sum > 0.f ? 1.0f / sum : 0.f;
      const uint32_t o_addr = tmem + ((uint32_t)(row & ~31) << 16) + 256 + 128 * t;
      const bool empty = range[t].j1 == 0;
#pragma unroll
      for (int c2 = 0; c2 < 4; ++c2) {
        float o[32];
        if (empty) {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0.f;
        } else tmem_ld32(o_addr + c2 * 32, o);
        if (row_valid) {
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) w[i >> 1] = pair_pack2<kBf16>(o[i] * inv, o[i + 1] * inv);
#pragma unroll
          for (int c = 0; c < 4; ++c)
            st16(out_row + (c2 * 4 + c) * 16, make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]));
        }
      }
    }
  }
  if (!ok && (tid & 31) == 0 && *(volatile int*)&sm->abort_flag == 0) { *(volatile int*)&sm->abort_flag = 1; report(p.status, TKV_DEV_TIMEOUT); }
  pair_finish<PfShape>(sm, tmem, k_issued, v_issued);
}

template <int kDtype>
static int launch_prefill(const CUtensorMap& mk, const CUtensorMap& mv, const AttnParams& p, int nseg, int nblocks,
                          cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(prefill_attn_kernel<kDtype>, cudaFuncAttributeMaxDynamicSharedMemorySize, PfShape::kBytes);
    if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_prefill_attn: %s", cudaGetErrorString(e));
    configured = true;
  }
  cudaError_t e = launch_pdl(prefill_attn_kernel<kDtype>, dim3((unsigned)((int64_t)nseg * nblocks)), dim3(kPairThreads),
                             (size_t)PfShape::kBytes, st, mk, mv, p, nseg, nblocks);
  if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_prefill_attn: %s", cudaGetErrorString(e));
  return check_launch("tkv_prefill_attn");
}

}  // namespace tkv

extern "C" int tkv_prefill_attn(const void* q, int64_t q_sb, int64_t q_st, int64_t q_sh,
                                const void* k_cache, const void* v_cache, const int32_t* seg_len, int64_t cap,
                                void* out, int batch, int hq, int hkv, int head_dim, int kv_dtype,
                                float scale, int max_len, int q_tokens, int32_t* status, tkv_stream_t stream) {
  using namespace tkv;
  if (!q || !k_cache || !v_cache || !out) return fail(TKV_ERR_ARG, "tkv_prefill_attn: NULL pointer argument");
  if (!(scale > 0.f)) return fail(TKV_ERR_ARG, "tkv_prefill_attn: scale must be positive");
  if (batch < 0 || hq <= 0 || hkv <= 0 || hq % hkv != 0 || max_len <= 0 || q_tokens < 1 || cap < max_len)
    return fail(TKV_ERR_ARG, "tkv_prefill_attn: bad sizes batch=%d hq=%d hkv=%d max_len=%d q_tokens=%d cap=%lld", batch, hq,
                hkv, max_len, q_tokens, (long long)cap);
  if (head_dim != 128 || (kv_dtype != TKV_BF16 && kv_dtype != TKV_F16))
    return fail(TKV_ERR_UNSUPPORTED, "tkv_prefill_attn: head_dim=%d dtype=%d (supported: 128, bf16/f16)", head_dim, kv_dtype);
  if (!aligned16(q) || !aligned16(k_cache) || !aligned16(v_cache) || !aligned16(out))
    return fail(TKV_ERR_ARG, "tkv_prefill_attn: pointers must be 16-byte aligned");
  if ((q_sb * 2) % 16 || (q_st * 2) % 16 || (q_sh * 2) % 16)
    return fail(TKV_ERR_ARG, "tkv_prefill_attn: q strides must be multiples of 16 bytes");
  if (batch == 0) return TKV_OK;
  const int nseg = batch * hkv, G = hq / hkv;
  const int64_t rows = (int64_t)q_tokens * G;
  const int64_t nblocks = (rows + kPfRows - 1) / kPfRows;
  if ((int64_t)nseg * nblocks > INT32_MAX || (int64_t)nseg * cap < kPfTile || (int64_t)nseg * cap + kPfTile > INT32_MAX)
    return fail(TKV_ERR_UNSUPPORTED, "tkv_prefill_attn: %lld query blocks x %d segments, %lld cache rows", (long long)nblocks,
                nseg, (long long)nseg * cap);
  AttnParams p;
  p.q = (const char*)q; p.q_sb = q_sb; p.q_sh = q_sh; p.q_st = q_st;
  p.k = (const char*)k_cache; p.v = (const char*)v_cache;
  p.seg_len = seg_len; p.seg_start = nullptr; p.cap = cap;
  p.out = (char*)out;
  p.part_ml = nullptr; p.part_o = nullptr; p.chunk = kPfTile; p.nchunks = 0;
  p.hq = hq; p.hkv = hkv; p.max_len = max_len;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  p.work = nullptr; p.work_count = nullptr; p.work_capacity = 0;
  p.q_tokens = q_tokens; p.rows = (int)rows;
  if (rows > INT32_MAX) return fail(TKV_ERR_UNSUPPORTED, "tkv_prefill_attn: too many query rows per segment");
  CUtensorMap mk, mv;
  int rc = make_map_2d(&mk, k_cache, 128, (int64_t)nseg * cap, 64, 128, kv_dtype);
  if (rc != TKV_OK) return rc;
  rc = make_map_2d(&mv, v_cache, 128, (int64_t)nseg * cap, 64, 128, kv_dtype);
  if (rc != TKV_OK) return rc;
  return kv_dtype == TKV_BF16 ? launch_prefill<TKV_BF16>(mk, mv, p, nseg, (int)nblocks, (cudaStream_t)stream)
                              : launch_prefill<TKV_F16>(mk, mv, p, nseg, (int)nblocks, (cudaStream_t)stream);
}
