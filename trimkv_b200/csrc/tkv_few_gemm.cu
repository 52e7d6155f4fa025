// Dense product of a few rows, out[m <= 16, n] = x[m, k] . w[n, k]^T in bf16, for the projections of a decoding step: HBM bounds
// it, and at these sizes (8 to 40 MB of weights) what counts is how soon all of the weights are on their way.
//
// One CTA per 16 or 32 rows of w, eight warps that split k; the warps' parts are added in warp order.  A lane copies the 16-byte
// pieces of its own fragments of m16n8k16 (a product does not mind in which order k is walked if both operands agree) into places
// of its own in shared memory, so that no thread waits for another one.  The weights do not depend on the kernel before this one:
// their first copies start before the wait for it, under programmatic launch while it still runs.
//
// us for 8 rows, back to back with weights from HBM, against the library's product: n x k 2048 x 2048 2.6 / 7.0, 2048 x 6144
// 6.4 / 16.2, 4224 x 2048 4.4 / 7.7, 8192 x 2048 6.3 / 8.2 (5.3 TB/s), 14336 x 2048 11.9 / 12.1; for 16 rows 3.1 / 5.6, 7.3 / 10.6,
// 5.1 / 6.3, 7.3 / 8.5, 13.6 / 12.3.
#include "tkv_elem.cuh"

namespace tkv {

constexpr int kFgWarps = 8, kFgThreads = kFgWarps * 32, kFgMost = 16;
// NT: tiles of eight rows of x, RT: tiles of 16 rows of w.  kAhead: steps (32 of k) a warp has on their way; two CTAs per SM.
template <int NT, int RT> struct FgRing {
  static constexpr int kPieces = 2 * RT + NT, kFit = 112 * 1024 / (kFgWarps * kPieces * 512), kAhead = kFit < 8 ? kFit : 8;
  static constexpr int kBytes = kFgWarps * kAhead * kPieces * 512, kRows = 16 * RT;
};

__device__ __forceinline__ void fg_mma(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void fg_copy(uint32_t dst, const __nv_bfloat16* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int NT, int RT>
__global__ void __launch_bounds__(kFgThreads, 2) few_gemm_kernel(const __nv_bfloat16* x, int64_t x_stride, const __nv_bfloat16* w, __nv_bfloat16* out,
                                                                int64_t out_stride, int m, int n, int k) {
  using R = FgRing<NT, RT>;
  extern __shared__ __align__(16) uint8_t ring[];                      // [warp][step][piece][lane] of 16 bytes, then the parts
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int row0 = blockIdx.x * R::kRows;
  const int steps = (k + 31) / 32, s0 = (int)((int64_t)warp * steps / kFgWarps), s1 = (int)((int64_t)(warp + 1) * steps / kFgWarps);
  // rows that do not exist repeat the last one: a row of either operand reaches only its own results, and those are not stored
  const __nv_bfloat16* wr[2 * RT];
#pragma unroll
  for (int r = 0; r < 2 * RT; ++r) wr[r] = w + (int64_t)min(row0 + g + 8 * r, n - 1) * k + c * 8;
  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) xr[t] = x + (int64_t)min(t * 8 + g, m - 1) * x_stride + c * 8;
  const uint32_t start = (uint32_t)__cvta_generic_to_shared(ring), mine = (uint32_t)(warp * R::kAhead * R::kPieces * 512 + lane * 16);
  auto place = [&](int s) { return mine + (uint32_t)((s - s0) % R::kAhead * R::kPieces * 512); };
  auto live = [&](int s) { return s * 32 + c * 8 < k; };               // k is whole pieces of 8: its last step may lack some, zeros then
  auto fetch_w = [&](int s) {
    if (s >= s1) return;
    const int at = live(s) ? s * 32 : -c * 8, bytes = live(s) ? 16 : 0;
#pragma unroll
    for (int r = 0; r < 2 * RT; ++r) fg_copy(start + place(s) + r * 512, wr[r] + at, bytes);
  };
  auto fetch_x = [&](int s) {
    if (s >= s1) return;
    const int at = live(s) ? s * 32 : -c * 8, bytes = live(s) ? 16 : 0;
#pragma unroll
    for (int t = 0; t < NT; ++t) fg_copy(start + place(s) + (2 * RT + t) * 512, xr[t] + at, bytes);
  };
#pragma unroll
  for (int u = 0; u < R::kAhead; ++u) fetch_w(s0 + u);                 // these belong to the first group
  grid_dependency_wait();
  grid_launch_dependents();
#pragma unroll
  for (int u = 0; u < R::kAhead; ++u) {
    fetch_x(s0 + u);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[NT][RT][4] = {};
  for (int s = s0; s < s1; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(R::kAhead - 1) : "memory");
    const uint4* at = reinterpret_cast<const uint4*>(ring + place(s));
    uint4 b[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) b[t] = at[32 * (2 * RT + t)];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const uint4 a0 = at[64 * r], a1 = at[64 * r + 32];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        fg_mma(acc[t][r], a0.x, a1.x, a0.y, a1.y, b[t].x, b[t].y);
        fg_mma(acc[t][r], a0.z, a1.z, a0.w, a1.w, b[t].z, b[t].w);
      }
    }
    fetch_w(s + R::kAhead);
    fetch_x(s + R::kAhead);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                                     // everyone has read its pieces: the parts take their place
  constexpr int kPitch = R::kRows + 1;
  static_assert(kFgWarps * NT * 8 * kPitch * 4 <= R::kBytes, "the parts take the place of the pieces");
  float* part = reinterpret_cast<float*>(ring);                        // [warp][row of x][kPitch]
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        part[(warp * NT * 8 + t * 8 + 2 * c + (i & 1)) * kPitch + 16 * r + g + 8 * (i >> 1)] = acc[t][r][i];
  __syncthreads();
  for (int i = tid; i < NT * 8 * R::kRows; i += kFgThreads) {
    const int t = i / R::kRows, row = i - t * R::kRows;
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < kFgWarps; ++j) v += part[(j * NT * 8 + t) * kPitch + row];
    if (t < m && row0 + row < n) out[(int64_t)t * out_stride + row0 + row] = __float2bfloat16_rn(v);
  }
}

template <int NT, int RT>
static int launch_few(const void* x, int64_t x_stride, const void* w, void* out, int64_t out_stride, int m, int n, int k, cudaStream_t st) {
  using R = FgRing<NT, RT>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(few_gemm_kernel<NT, RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, R::kBytes);
    if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_few_gemm: %s", cudaGetErrorString(e));
    configured = true;
  }
  cudaError_t e = launch_pdl(few_gemm_kernel<NT, RT>, dim3((n + R::kRows - 1) / R::kRows), dim3(kFgThreads), (size_t)R::kBytes, st,
                             (const __nv_bfloat16*)x, x_stride, (const __nv_bfloat16*)w, (__nv_bfloat16*)out, out_stride, m, n, k);
  if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_few_gemm: %s", cudaGetErrorString(e));
  return check_launch("tkv_few_gemm");
}
// 32 rows of w per CTA once 16 would give more CTAs than the SMs hold at a time: x is then read half as often (8192 x 2048, 8 rows:
// 8.4 us with 16, 6.3 us with 32).
template <int NT>
static int launch_few(const void* x, int64_t x_stride, const void* w, void* out, int64_t out_stride, int m, int n, int k, cudaStream_t st) {
  return n > 2 * 148 * 16 ? launch_few<NT, 2>(x, x_stride, w, out, out_stride, m, n, k, st) : launch_few<NT, 1>(x, x_stride, w, out, out_stride, m, n, k, st);
}

}  // namespace tkv

extern "C" int tkv_few_gemm(const void* x, int64_t x_stride, const void* w, void* out, int64_t out_stride, int m, int n, int k, int dtype,
                            tkv_stream_t stream) {
  using namespace tkv;
  if (!x || !w || !out) return fail(TKV_ERR_ARG, "tkv_few_gemm: NULL pointer argument");
  if (m <= 0 || n <= 0 || k <= 0 || x_stride < k || out_stride < n) return fail(TKV_ERR_ARG, "tkv_few_gemm: bad sizes m=%d n=%d k=%d", m, n, k);
  if (dtype != TKV_BF16 || m > kFgMost || k % 8 || x_stride % 8 || !aligned16(x) || !aligned16(w))
    return fail(TKV_ERR_UNSUPPORTED, "tkv_few_gemm: up to %d bf16 rows of whole 16-byte pieces (m=%d k=%d)", kFgMost, m, k);
  cudaStream_t st = (cudaStream_t)stream;
  return m <= 8 ? launch_few<1>(x, x_stride, w, out, out_stride, m, n, k, st) : launch_few<2>(x, x_stride, w, out, out_stride, m, n, k, st);
}
