// Windowed differential attention over many query tokens (prompts and portions of prompts) on tcgen05 + TMEM.
//
// One CTA = (request, kv head, block of 128 query rows), row = token * heads_per_kv + head, on the core of tkv_attn_pair.cuh:
// its two tiles are the two maps of the same rows, each with queries and keys of its own; a V tile is loaded once for both.  The
// epilogue combines the maps, norms the head and applies the gate in fp32 registers: nothing of a map's output goes to memory.
// A row sees the columns [lo, hi) of the request's linear keys; tiles before the first row's window are never loaded.  Waits are
// bounded; on expiry the CTA records TKV_DEV_TIMEOUT, drains its copies and frees its TMEM.
#include <cuda.h>
#include "tkv_attn_pair.cuh"
#include "tkv_diffattn.cuh"

namespace tkv {

// KH = dp / 64, VH = pp / 64.  Warpgroup m: softmax of map m; in the epilogue half m of a row's dims.
template <int KH, int VH>
__global__ void __launch_bounds__(kPairThreads, 1)
diff_prefill_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, DiffAttnParams p, int nblocks) {
  extern __shared__ __align__(1024) uint8_t base[];
  using Shape = PairShape<KH, VH, true>;
  constexpr int DP = KH * 64, PP = VH * 64;
  constexpr int OD = PP / 2;                               // dims of O per thread in the epilogue: 32 or 64
  grid_dependency_wait();
  grid_launch_dependents();
  const int seg = (int)(blockIdx.x / (unsigned)nblocks);
  const int blk = nblocks - 1 - (int)(blockIdx.x % (unsigned)nblocks);
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5);
  const bool is_row = warp < 8;
  const int row = tid & (kDaTile - 1), half = (tid >> 7) & 1;
  const int hpg = p.heads / p.kv_heads;
  const int b = seg / p.kv_heads, g = seg - b * p.kv_heads;
  const int tok0 = p.cu[b], n = p.cu[b + 1] - tok0;
  const int rows = n * hpg;
  if (blk * kDaTile >= rows) return;
  if ((smem_u32(base) & 1023u) != 0) {                     // the swizzled tiles need it; the launch gives it
    if (tid == 0) report(p.status, TKV_DEV_TIMEOUT);
    return;
  }
  const int hist = min(p.pos0[b], p.window - 1);
  const int len = hist + n;                                // linear rows of the request
  const int R = blk * kDaTile + row;
  const bool row_valid = is_row && R < rows;
  const int token = row_valid ? R / hpg : 0, head = g * hpg + (row_valid ? R - token * hpg : 0);
  const int hi_row = row_valid ? hist + token + 1 : 0, lo_row = max(0, hi_row - p.window);
  const int hi_max = hist + (min(blk * kDaTile + kDaTile, rows) - 1) / hpg + 1;
  const int lo_min = max(0, hist + (blk * kDaTile) / hpg + 1 - p.window);
  const int tile0 = lo_min / kDaTile, ntiles = (hi_max + kDaTile - 1) / kDaTile - tile0;
  const PairRange range[2] = {{0, ntiles}, {0, ntiles}};
  const int kv0 = p.kv_start[b] + tile0 * kDaTile;

  PairSmem* sm = Shape::smem(base);
  if (tid == 0) pair_init(sm);
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)), "r"(kDaTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  } else if (is_row) {
    const __nv_bfloat16* qp = (const __nv_bfloat16*)p.q + (((int64_t)(tok0 + token) * p.heads + head) * 2 + half) * DP;
    uint8_t* q_s = Shape::q(base, half);
#pragma unroll
    for (int c = 0; c < DP / 8; ++c) st16(q_s + da_swz(row, c), row_valid ? ld16(qp + c * 8) : make_uint4(0, 0, 0, 0));
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;

  int k_issued = 0, v_issued = 0;
  bool ok = true;
  if (warp == 8) {
    ok = pair_products<Shape, true>(sm, base, tmem, ntiles, range);
    __syncwarp();
  } else if (warp == 9) {
    if ((tid & 31) == 0)
      ok = pair_copies<Shape>(sm, ntiles,
          [&](int j) {
#pragma unroll
            for (int i = 0; i < 2 * KH; ++i)               // map i / KH
              tma_load_2d(Shape::k(base, j) + i * kDaHalf, &map_k, &sm->full_k[j % Shape::kNK], g * 2 * DP + i * 64, kv0 + j * kDaTile);
          },
          [&](int j) {
#pragma unroll
            for (int i = 0; i < VH; ++i)
              tma_load_2d(Shape::v(base, j) + i * kDaHalf, &map_v, &sm->full_v[j % Shape::kNV], g * PP + i * 64, kv0 + j * kDaTile);
          }, &k_issued, &v_issued);
    __syncwarp();
  } else {
    float sum = 0.f;
    ok = pair_softmax<Shape, true, false>(sm, base, tmem, half, range[half], lo_row, hi_row, tile0 * kDaTile, len, p.scale_log2, &sum);
    // ---- epilogue: both maps / their sums, combination, norm over the head (two threads per row), gate
    if (ok) {
      sm->red[half][row] = sum;
      tc_fence_before();
      ok = pair_meet(sm, 0);                               // the other map's output is complete as well
    }
    if (ok) {
      tc_fence_after();
      const uint32_t lane_base = tmem + ((uint32_t)(row & ~31) << 16);
      const float l0 = sm->red[0][row], l1 = sm->red[1][row];
      const float i0 = l0 > 0.f ? 1.0f / l0 : 0.f, i1 = l1 > 0.f ? *p.lambda / l1 : 0.f;
      float o[OD], ss = 0.f;
#pragma unroll
      for (int c2 = 0; c2 < OD / 32; ++c2) {
        float x[32];
        tmem_ld32(lane_base + 256 + OD * half + c2 * 32, o + c2 * 32);
        tmem_ld32(lane_base + 384 + OD * half + c2 * 32, x);
#pragma unroll
        for (int i = 0; i < 32; ++i) {                     // padded dims are zero in both maps
          o[c2 * 32 + i] = o[c2 * 32 + i] * i0 - x[i] * i1;
          ss += o[c2 * 32 + i] * o[c2 * 32 + i];
        }
      }
      float* xch = reinterpret_cast<float*>(base);         // every product that read Q has completed
      xch[half * kDaTile + row] = ss;
      ok = pair_meet(sm, 1);
      if (ok && row_valid) {
        const float rr = 1.0f / sqrtf((ss + xch[(half ^ 1) * kDaTile + row]) / (float)p.vdim + p.eps);
        const float gate = rr * (1.0f - p.diff) *
                           sigmoid_f32(__bfloat162float(((const __nv_bfloat16*)p.gate)[(int64_t)(tok0 + token) * p.gate_stride + head]));
        __nv_bfloat16* dst = (__nv_bfloat16*)p.out + ((int64_t)(tok0 + token) * p.heads + head) * p.vdim + half * OD;
        const int live = min(OD, p.vdim - half * OD);      // dims of this thread that exist
        if (p.vdim % 8 == 0) {
#pragma unroll
          for (int i = 0; i < OD; i += 8)
            if (i < live)
              st16(dst + i, make_uint4(da_pack2(o[i] * gate, o[i + 1] * gate), da_pack2(o[i + 2] * gate, o[i + 3] * gate),
                                       da_pack2(o[i + 4] * gate, o[i + 5] * gate), da_pack2(o[i + 6] * gate, o[i + 7] * gate)));
        } else {
#pragma unroll
          for (int i = 0; i < OD; ++i)
            if (i < live) dst[i] = __float2bfloat16_rn(o[i] * gate);
        }
      }
    }
  }
  if (!ok && (tid & 31) == 0 && *(volatile int*)&sm->abort_flag == 0) { *(volatile int*)&sm->abort_flag = 1; report(p.status, TKV_DEV_TIMEOUT); }
  pair_finish<Shape>(sm, tmem, k_issued, v_issued);
}

template <int KH, int VH>
static int launch_da(const CUtensorMap& mk, const CUtensorMap& mv, const DiffAttnParams& p, int64_t grid, int nblocks, cudaStream_t st) {
  static bool configured = false;
  constexpr int kBytes = PairShape<KH, VH, true>::kBytes;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(diff_prefill_kernel<KH, VH>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_diff_prefill: %s", cudaGetErrorString(e));
    configured = true;
  }
  cudaError_t e = launch_pdl(diff_prefill_kernel<KH, VH>, dim3((unsigned)grid), dim3(kPairThreads), (size_t)kBytes, st, mk, mv, p, nblocks);
  if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_diff_prefill: %s", cudaGetErrorString(e));
  return check_launch("tkv_diff_prefill");
}

int launch_diff_prefill_tc(const DiffAttnParams& p, int64_t kv_rows, int max_tokens, cudaStream_t st) {
  const int64_t rows = (int64_t)max_tokens * (p.heads / p.kv_heads), nblocks = (rows + kDaTile - 1) / kDaTile;
  const int64_t grid = (int64_t)p.batch * p.kv_heads * nblocks;
  if (grid > INT32_MAX || rows > INT32_MAX - kDaTile || kv_rows + kDaTile > INT32_MAX)
    return fail(TKV_ERR_UNSUPPORTED, "tkv_diff_prefill: %lld query blocks, %lld key rows", (long long)grid, (long long)kv_rows);
  if (!aligned16(p.q) || !aligned16(p.k_lin) || !aligned16(p.v_lin) || !aligned16(p.out))
    return fail(TKV_ERR_ARG, "tkv_diff_prefill: pointers must be 16-byte aligned");
  CUtensorMap mk, mv;
  int rc = make_map_2d(&mk, p.k_lin, (int64_t)p.kv_heads * 2 * p.dp, kv_rows, 64, 128, TKV_BF16);
  if (rc != TKV_OK) return rc;
  rc = make_map_2d(&mv, p.v_lin, (int64_t)p.kv_heads * p.pp, kv_rows, 64, 128, TKV_BF16);
  if (rc != TKV_OK) return rc;
  if (p.dp == 64) return p.pp == 64 ? launch_da<1, 1>(mk, mv, p, grid, (int)nblocks, st) : launch_da<1, 2>(mk, mv, p, grid, (int)nblocks, st);
  return p.pp == 64 ? launch_da<2, 1>(mk, mv, p, grid, (int)nblocks, st) : launch_da<2, 2>(mk, mv, p, grid, (int)nblocks, st);
}

}  // namespace tkv
