// Product of a few rows: y[m <= 32, n] = x[m, k] . w[n, k]^T + bias[n] in bf16, on tcgen05 with TMA.
//
// What bounds it is the stream of the weights, and for 4 to 40 MB of them the time until the stream runs and after it ends.  128 rows
// of w are the products' M, the rows of x their N; k is divided among the CTAs of a cluster, so that a product of few columns has
// every SM stream, and their sums meet in shared memory, in the order of k: no partial sums in memory and no second kernel.
// A stage costs its copies' warp some 500 cycles whatever it holds: stages of 16 KB of weights stream 56 GB/s into an SM, of 32 KB, one
// copy each for w and x, 81.  Five of those fill an SM.
// What does not depend on the kernel before, the weights, is asked for before its end is waited for, into L2 only: a copy into L2
// is right even if that kernel should write them.
//   warp 0  copies: 128 columns of w and x a stage     warp 1  products into 32 (16) columns of TMEM
//   all     TMEM -> shared memory [row of x][row of w]; cluster; then each CTA adds up its share of the rows of x and stores
// us in a replayed graph, each behind an elementwise kernel of 2 to 3 us on x, library and this, for 8 rows, 32 rows:
//   2048 x 2048  8.9 5.7, 7.4 6.4      2048 x 4096  13.0 7.3, 10.0 8.1      2048 x 9216  23.8 10.4, 16.3 11.8     4096 x 2048  9.6 6.3, 8.1 7.4
//   5120 x 2048  8.2 7.6, 9.3 8.7      9216 x 2048  10.6 10.0, 10.9 11.4    12288 x 2048 12.4 13.5, 13.9 14.6     32768 x 2048 27.4 29.3, 29.9 32.0
// Every wait is bounded; on expiry the CTA records TKV_DEV_TIMEOUT, gives zeros to its cluster, drains its copies and frees its TMEM.
#include "tkv_tc.cuh"

namespace tkv {

constexpr int kFrThreads = 128, kFrSubs = 2, kFrW = kFrSubs * 128 * 64 * 2;
template <int N> struct FrRing {
  static constexpr int kStage = kFrW + kFrSubs * N * 128, kStages = 5;
  static_assert(kStages * kStage >= N * 512, "the sums of a CTA take the place of the stages");
};
template <int S> struct FrSmemOf {
  uint64_t full[S], empty[S], done;
  uint32_t tmem_base;
  int abort_flag;
};
template <int N> using FrSmem = FrSmemOf<FrRing<N>::kStages>;
template <int N> constexpr int fr_smem_bytes() { return FrRing<N>::kStages * FrRing<N>::kStage + (int)sizeof(FrSmem<N>); }

struct FewRows {
  void* y; const __nv_bfloat16* bias;                      // bias [n] or NULL
  int m, n, pieces, splits;                                // pieces of 128 columns of k
  int32_t* status;
};

__device__ __forceinline__ float4 ld_cluster(uint32_t at, int rank) {
  float4 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at), "r"(rank) : "memory");
  return v;
}

template <int N>
__global__ void __launch_bounds__(kFrThreads)
few_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, FewRows p) {
  extern __shared__ __align__(1024) uint8_t base[];
  constexpr int S = FrRing<N>::kStages, kStage = FrRing<N>::kStage, kCols = 32;
  FrSmem<N>* sm = reinterpret_cast<FrSmem<N>*>(base + S * kStage);
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int tile = blockIdx.x / p.splits, rank = blockIdx.x - tile * p.splits;
  const int first = (int)((int64_t)rank * p.pieces / p.splits), steps = (int)((int64_t)(rank + 1) * p.pieces / p.splits) - first;
  volatile int* abort_flag = &sm->abort_flag;
  if (warp == 0) {
    if (elect_one())
      for (int i = 0; i < steps && i < S - 1; ++i)
        asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];" ::"l"(&map_w), "r"(0), "r"(tile * 128), "r"((first + i) * kFrSubs) : "memory");
    __syncwarp();
  }
  if (tid == 0) {
    for (int s = 0; s < S; ++s) { mbar_init(&sm->full[s], 1); mbar_init(&sm->empty[s], 1); }
    mbar_init(&sm->done, 1);
    sm->abort_flag = (smem_u32(base) & 1023u) != 0;        // the swizzled tiles need the alignment; the launch gives it
    if (sm->abort_flag) report(p.status, TKV_DEV_TIMEOUT);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)), "r"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;
  const bool sound = *abort_flag == 0;                     // one decision for the whole CTA
  grid_dependency_wait();
  grid_launch_dependents();
  int copies = 0;
  if (warp == 0) {
    bool ok = sound;
    for (int i = 0; i < steps && ok; ++i) {
      const int s = i % S;
      ok = warp_wait(&sm->empty[s], ((i / S) & 1) ^ 1, abort_flag);
      if (!ok) break;
      if (elect_one()) {
        uint8_t* st = base + s * kStage;
        mbar_expect_tx(&sm->full[s], kStage);
        tma_load_3d(st, &map_w, &sm->full[s], 0, tile * 128, (first + i) * kFrSubs);
        tma_load_3d(st + kFrW, &map_x, &sm->full[s], 0, 0, (first + i) * kFrSubs);
      }
      __syncwarp();
      ++copies;
    }
    if (!ok && lane == 0 && *abort_flag == 0) { *abort_flag = 1; report(p.status, TKV_DEV_TIMEOUT); }
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc(1, 0, N), tm = warp_uniform(tmem);
    const uint64_t w0 = make_desc(smem_u32(base), 16, 1024, 2);
    bool ok = sound;
    for (int i = 0; i < steps && ok; ++i) {
      const int s = i % S;
      ok = warp_wait(&sm->full[s], (i / S) & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t w = w0 + (uint32_t)s * (kStage >> 4);
#pragma unroll
        for (int q = 0; q < 4 * kFrSubs; ++q)
          umma(tm, w + (q >> 2) * 1024 + (q & 3) * 2, w + (kFrW >> 4) + (q >> 2) * (N * 8) + (q & 3) * 2, idesc, i > 0 || q > 0);
        umma_commit(&sm->empty[s]);
        if (i == steps - 1) umma_commit(&sm->done);
      }
      __syncwarp();
    }
    if (!ok && lane == 0 && *abort_flag == 0) { *abort_flag = 1; report(p.status, TKV_DEV_TIMEOUT); }
  }
  __syncwarp();
  if (sound && !mbar_wait_or_abort(&sm->done, 0, abort_flag) && *abort_flag == 0) { *abort_flag = 1; report(p.status, TKV_DEV_TIMEOUT); }
  __syncthreads();                                         // one decision for the whole CTA
  const bool have = *abort_flag == 0;
  if (!have) {                                             // copies in flight land before anything else is written there
    if (warp == 0)
      for (int i = max(0, copies - S); i < copies; ++i) mbar_wait(&sm->full[i % S], (i / S) & 1);
    __syncthreads();
  }
  tc_fence_after();
  float* const part = reinterpret_cast<float*>(base);      // [N][128]
  {
    float acc[32];
    if (have) {
      if constexpr (N == 16) tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16), acc);
      else tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16), acc);
    }
#pragma unroll
    for (int r = 0; r < N; ++r) part[r * 128 + tid] = have ? acc[r] : 0.f;
  }
  tc_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int col = tile * 128 + lane * 4;
  if (col < p.n)
    for (int r = rank * 4 + warp; r < p.m; r += 4 * p.splits) {
      const uint32_t at = smem_u32(part + r * 128 + lane * 4);
      float4 sum = ld_cluster(at, 0);
      for (int c = 1; c < p.splits; ++c) {
        const float4 v = ld_cluster(at, c);
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
      }
      if (p.bias != nullptr) {
        const uint2 b = *reinterpret_cast<const uint2*>(p.bias + col);
        sum.x += __uint_as_float(b.x << 16); sum.y += __uint_as_float(b.x & 0xffff0000u);
        sum.z += __uint_as_float(b.y << 16); sum.w += __uint_as_float(b.y & 0xffff0000u);
      }
      const int64_t to = (int64_t)r * p.n + col;
      const __nv_bfloat162 lo = __floats2bfloat162_rn(sum.x, sum.y), hi = __floats2bfloat162_rn(sum.z, sum.w);
      *reinterpret_cast<uint2*>((__nv_bfloat16*)p.y + to) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");    // nobody reads this CTA's sums any more
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
}

// CTAs along k: clusters of s, a CTA to an SM, run room[s] at a time (148, 74, 45, 33, 26, 22, 15, 15 of 1 to 8 CTAs on a B200: clusters of eight leave 28
// SMs idle); a wave of them costs its pieces and about six more until they arrive and after they have been added up.
static int few_rows_splits(const int* room, int tiles, int pieces) {
  int best = 1; long cost = -1;
  for (int s = 1; s <= 8 && s <= pieces; ++s) {
    if (room[s] < 1) continue;
    const long c = (long)((tiles + room[s] - 1) / room[s]) * ((pieces + s - 1) / s + 6);
    if (cost < 0 || c < cost) { best = s; cost = c; }
  }
  return best;
}

template <int N>
static int launch_few_rows(const void* x, const void* w, FewRows p, int k, cudaStream_t st) {
  CUtensorMap mw, mx;
  int rc = make_map_pieces(&mw, w, k, p.n, 128, kFrSubs);
  if (rc == TKV_OK) rc = make_map_pieces(&mx, x, k, p.m, N, kFrSubs);
  if (rc != TKV_OK) return rc;
  const int bytes = fr_smem_bytes<N>();
  static int room[9];
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.blockDim = dim3(kFrThreads); cfg.dynamicSmemBytes = bytes; cfg.stream = st; cfg.attrs = attr;
  if (room[1] == 0) {
    cudaError_t e = cudaFuncSetAttribute(few_rows_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_few_rows: %s", cudaGetErrorString(e));
    for (int s = 8; s >= 1; --s) {
      attr[0].val.clusterDim.x = (unsigned)s; cfg.gridDim = dim3((unsigned)s * 148); cfg.numAttrs = 1;
      cudaOccupancyMaxActiveClusters(&room[s], few_rows_kernel<N>, &cfg);
    }
  }
  const int tiles = (p.n + 127) / 128;
  p.splits = few_rows_splits(room, tiles, p.pieces);
  attr[0].val.clusterDim.x = (unsigned)p.splits; cfg.gridDim = dim3((unsigned)(tiles * p.splits)); cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, few_rows_kernel<N>, mw, mx, p);
  if (e != cudaSuccess) return fail(TKV_ERR_LAUNCH, "tkv_few_rows: %s", cudaGetErrorString(e));
  return check_launch("tkv_few_rows");
}

}  // namespace tkv

extern "C" int tkv_few_rows(const void* x, const void* w, const void* bias, void* y, int m, int n, int k, int32_t* status, tkv_stream_t stream) {
  using namespace tkv;
  if (!x || !w || !y) return fail(TKV_ERR_ARG, "tkv_few_rows: NULL pointer argument");
  if (m <= 0 || m > 32 || n <= 0 || k <= 0 || n % 8 || k % 64)
    return fail(TKV_ERR_UNSUPPORTED, "tkv_few_rows: m=%d n=%d k=%d (supported: m <= 32, n %% 8 == 0, k %% 64 == 0)", m, n, k);
  if (!aligned16(x) || !aligned16(w) || !aligned16(y) || (bias && !aligned16(bias))) return fail(TKV_ERR_ARG, "tkv_few_rows: pointers must be 16-byte aligned");
  FewRows p = {};
  p.y = y; p.bias = (const __nv_bfloat16*)bias; p.m = m; p.n = n; p.pieces = (k / 64 + kFrSubs - 1) / kFrSubs; p.status = status;
  return m <= 16 ? launch_few_rows<16>(x, w, p, k, (cudaStream_t)stream) : launch_few_rows<32>(x, w, p, k, (cudaStream_t)stream);
}
