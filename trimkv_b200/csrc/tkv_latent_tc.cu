// Windowed attention with keys in two parts over many query tokens (prompts and portions of prompts) on tcgen05 + TMEM.
//
// One CTA = (request, head, block of 256 query tokens) as two tiles of 128 rows on the core of tkv_attn_pair.cuh; a key tile is
// fetched as 64-column pieces, the first part from the head's keys, the second from the row that all heads share.  Pieces beyond
// a part's width are zero-filled by the copy.  A row sees the columns [lo, hi) of the request's linear keys; a tile's key range
// goes from its first row's window to its last row.  Waits are bounded; on expiry the CTA records TKV_DEV_TIMEOUT, drains its
// copies and frees its TMEM.
#include <cuda.h>
#include "tkv_attn_pair.cuh"
#include "tkv_latent.cuh"

namespace tkv {

constexpr int kTpRows = 2 * kDaTile;                       // query tokens per CTA

// K1, K2: 64-element pieces of the two key parts; VH: of a value.
template <int K1, int K2, int VH>
__global__ void __launch_bounds__(kPairThreads, 1)
two_part_prefill_kernel(const __grid_constant__ CUtensorMap map_k1, const __grid_constant__ CUtensorMap map_k2,
                        const __grid_constant__ CUtensorMap map_v, TwoPartAttn p, int nblocks) {
  extern __shared__ __align__(1024) uint8_t base[];
  constexpr int KH = K1 + K2;
  using Shape = PairShape<KH, VH, false>;
  grid_dependency_wait();
  grid_launch_dependents();
  const int seg = (int)(blockIdx.x / (unsigned)nblocks);
  const int blk = nblocks - 1 - (int)(blockIdx.x % (unsigned)nblocks);
  const int tid = threadIdx.x, warp = tid >> 5;
  const bool is_row = warp < 8;
  const int row = tid & (kDaTile - 1), t = (tid >> 7) & 1;
  const int b = seg / p.heads, head = seg - b * p.heads;
  const int tok0 = p.cu[b], n = p.cu[b + 1] - tok0;
  if (blk * kTpRows >= n) return;
  if ((smem_u32(base) & 1023u) != 0) {                     // the swizzled tiles need it; the launch gives it
    if (tid == 0) report(p.status, TKV_DEV_TIMEOUT);
    return;
  }
  const int hist = min(p.pos0[b], p.window - 1);
  const int len = hist + n;                                // linear rows of the request
  const int R = blk * kTpRows + t * kDaTile + row;
  const bool row_valid = is_row && R < n;
  const int token = row_valid ? R : 0;
  const int hi_row = row_valid ? hist + token + 1 : 0, lo_row = max(0, hi_row - p.window);
  const int tile0 = max(0, hist + blk * kTpRows + 1 - p.window) / kDaTile;
  PairRange range[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int first = blk * kTpRows + i * kDaTile, last = min(first + kDaTile, n);
    range[i] = {max(0, hist + first + 1 - p.window) / kDaTile - tile0, (hist + last + kDaTile - 1) / kDaTile - tile0};
    if (first >= n) range[i] = {0, 0};
  }
  const int ntiles = max(range[0].j1, range[1].j1);
  const float scale_log2 = p.scale * 1.4426950408889634f;
  const int kv0 = p.kv_start[b] + tile0 * kDaTile;

  PairSmem* sm = Shape::smem(base);
  if (tid == 0) pair_init(sm);
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)), "r"(kDaTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  } else if (is_row && range[t].j1 > 0) {
    const __nv_bfloat16* q1 = (const __nv_bfloat16*)p.q1 + (int64_t)(tok0 + token) * p.q1_token + (int64_t)head * p.q1_head;
    const __nv_bfloat16* q2 = (const __nv_bfloat16*)p.q2 + (int64_t)(tok0 + token) * p.q2_token + (int64_t)head * p.q2_head;
    uint8_t* q_s = Shape::q(base, t);
#pragma unroll
    for (int c = 0; c < KH * 8; ++c) {
      const bool first = c < K1 * 8;
      const int e = (first ? c : c - K1 * 8) * 8;
      const bool live = row_valid && e < (first ? p.d1 : p.d2);
      st16(q_s + da_swz(row, c), live ? ld16((first ? q1 : q2) + e) : make_uint4(0, 0, 0, 0));
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;

  int k_issued = 0, v_issued = 0;
  bool ok = true;
  if (warp == 8) {
    if ((tid & 31) == 0) ok = pair_products<Shape, true>(sm, base, tmem, ntiles, range);
    __syncwarp();
  } else if (warp == 9) {
    if ((tid & 31) == 0)
      ok = pair_copies<Shape>(sm, ntiles,
          [&](int j) {
            uint64_t* bar = &sm->full_k[j % Shape::kNK];
#pragma unroll
            for (int i = 0; i < K1; ++i) tma_load_3d(Shape::k(base, j) + i * kDaHalf, &map_k1, bar, i * 64, head, kv0 + j * kDaTile);
#pragma unroll
            for (int i = 0; i < K2; ++i) tma_load_3d(Shape::k(base, j) + (K1 + i) * kDaHalf, &map_k2, bar, i * 64, 0, kv0 + j * kDaTile);
          },
          [&](int j) {
#pragma unroll
            for (int i = 0; i < VH; ++i)
              tma_load_3d(Shape::v(base, j) + i * kDaHalf, &map_v, &sm->full_v[j % Shape::kNV], i * 64, head, kv0 + j * kDaTile);
          }, &k_issued, &v_issued);
    __syncwarp();
  } else {
    float l = 0.f;
    ok = pair_softmax<Shape, true, true>(sm, base, tmem, t, range[t], lo_row, hi_row, tile0 * kDaTile, len, scale_log2, &l);
    if (ok && range[t].j1 > 0) {                           // a tile without rows has nothing to write
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      const uint32_t o_addr = tmem + ((uint32_t)(row & ~31) << 16) + 256 + 128 * t;
      __nv_bfloat16* dst = (__nv_bfloat16*)p.out + (int64_t)(tok0 + token) * p.out_token + (int64_t)head * p.out_head;
#pragma unroll
      for (int c2 = 0; c2 < 2 * VH; ++c2) {
        float o[32];
        tmem_ld32(o_addr + c2 * 32, o);
        if (row_valid)
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            if (c2 * 32 + i < p.vdim)
              st16(dst + c2 * 32 + i, make_uint4(da_pack2(o[i] * inv, o[i + 1] * inv), da_pack2(o[i + 2] * inv, o[i + 3] * inv),
                                                 da_pack2(o[i + 4] * inv, o[i + 5] * inv), da_pack2(o[i + 6] * inv, o[i + 7] * inv)));
      }
    }
  }
  if (!ok && (tid & 31) == 0 && *(volatile int*)&sm->abort_flag == 0) { *(volatile int*)&sm->abort_flag = 1; report(p.status, TKV_DEV_TIMEOUT); }
  pair_finish<Shape>(sm, tmem, k_issued, v_issued);
}

// Parts of whole 16-byte pieces: every row, head and part starts on a 16-byte boundary.
bool two_part_tc_shape(const TwoPartAttn& p, int dtype) {
  if (dtype != TKV_BF16 || p.ring_rows > 0 || p.scale <= 0.f) return false;
  if (p.d1 > 128 || p.d2 <= 0 || p.d2 > 64 || p.vdim > 128 || p.d1 % 8 || p.d2 % 8 || p.vdim % 8) return false;
  if (p.q1_token % 8 || p.q2_token % 8 || p.k1_row % 8 || p.k2_row % 8 || p.v_row % 8 || p.out_token % 8) return false;
  return aligned16(p.q1) && aligned16(p.q2) && aligned16(p.k1) && aligned16(p.k2) && aligned16(p.v) && aligned16(p.out);
}

template <int K1, int VH>
static int launch_tp(const CUtensorMap& m1, const CUtensorMap& m2, const CUtensorMap& mv, const TwoPartAttn& p, int64_t grid, int nblocks,
                     cudaStream_t st) {
  static bool configured = false;
  constexpr int kBytes = PairShape<K1 + 1, VH, false>::kBytes;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(two_part_prefill_kernel<K1, 1, VH>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_latent_prefill: %s", cudaGetErrorString(e));
    configured = true;
  }
  cudaError_t e = launch_pdl(two_part_prefill_kernel<K1, 1, VH>, dim3((unsigned)grid), dim3(kPairThreads), (size_t)kBytes, st, m1, m2, mv, p, nblocks);
  if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_latent_prefill: %s", cudaGetErrorString(e));
  return check_launch("tkv_latent_prefill");
}

int launch_two_part_tc(const TwoPartAttn& p, int64_t kv_rows, int max_tokens, cudaStream_t st) {
  const int64_t nblocks = ((int64_t)max_tokens + kTpRows - 1) / kTpRows, grid = (int64_t)p.batch * p.heads * nblocks;
  if (grid > INT32_MAX || kv_rows + kDaTile > INT32_MAX)
    return fail(TKV_ERR_UNSUPPORTED, "tkv_latent_prefill: %lld query blocks, %lld key rows", (long long)grid, (long long)kv_rows);
  CUtensorMap m1, m2, mv;
  int rc = make_map_3d_bf16(&m1, p.k1, p.d1, p.heads, kv_rows, p.k1_row, 64, 128);
  if (rc == TKV_OK) rc = make_map_3d_bf16(&m2, p.k2, 64, 1, kv_rows, p.k2_row, 64, 128);
  if (rc == TKV_OK) rc = make_map_3d_bf16(&mv, p.v, p.vdim, p.heads, kv_rows, p.v_row, 64, 128);
  if (rc != TKV_OK) return rc;
  if (p.d1 <= 64) return p.vdim <= 64 ? launch_tp<1, 1>(m1, m2, mv, p, grid, (int)nblocks, st) : launch_tp<1, 2>(m1, m2, mv, p, grid, (int)nblocks, st);
  return p.vdim <= 64 ? launch_tp<2, 1>(m1, m2, mv, p, grid, (int)nblocks, st) : launch_tp<2, 2>(m1, m2, mv, p, grid, (int)nblocks, st);
}

}  // namespace tkv
