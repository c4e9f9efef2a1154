// float64 matrix multiply on the double-precision matrix instruction (mma.sync m8n8k4; tcgen05 has no
// 64-bit kind). Row-major operands with leading dimensions, either operand transposed, batched with
// strides, the same fused epilogue as the other products.
//
// What bounds it: the FP64 units, 64 fused multiply-adds per clock and SM (about 36 TFLOP/s), once the
// operands arrive early enough. Tiles of 64 x 64 (or 32 x 32 where 64 x 64 would leave SMs without one)
// are multiplied by four warps; 16-deep k slabs travel through a four-stage cp.async ring in whichever
// order they are stored, so neither transposed operand needs a pass of its own. A matrix instruction
// reads one value of A and one of B per lane for 256 multiply-adds, where the scalar kernel this
// replaces read eight values through shared memory for sixteen.
// Row pitches in shared memory are 4 (mod 16) doubles: the 4 x 4 (row, k) lanes of half a warp then fall
// into 16 distinct 8-byte banks in either storage order.
//
// Products with too few tiles for the GPU are cut along k as well. Each block leaves its partial tile in
// arena scratch and the one that arrives last adds the parts in k order, so a result does not depend on
// which block that was; no block waits for another.
//
// Measured (B200, kernel alone): 256 x 300 x 784 316 -> 17 us, 256 x 784 x 300 (B transposed)
// 110 -> 14 us, 784 x 300 x 256 (A transposed) 99 -> 14 us.
#include <algorithm>
#include <atomic>

#include "engine.h"
#include "epilogue.cuh"
#include "ptx.cuh"

namespace b200 {

constexpr int F64_BK = 16, F64_STAGES = 4, F64_THREADS = 128;

struct GemmF64Params {
  long long M, N, K;
  const double *A, *B;
  double *C;
  long long lda, ldb, ldc, strideA, strideB, strideC;
  int tiles_n, splits;
  double *ws;       // partial tiles, [batch][tile][split], when splits > 1
  int *tile_count;  // parts delivered per (batch, tile); zero between launches
  Epilogue ep;
};

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
// Copies V doubles, of which the first `valid` exist; the rest arrive as zeros.
template <int V>
__device__ __forceinline__ void cp_async_f64(double *dst, const double *src, int valid) {
  if (V == 2)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_addr(dst)), "l"(src), "r"(valid * 8)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(ptx::smem_addr(dst)), "l"(src), "r"(valid * 8)
                 : "memory");
}

// One operand's slab: T rows/columns of the tile by F64_BK of k. MN: stored with m (n) contiguous.
template <int T, bool MN>
struct SlabF64 {
  static constexpr int PITCH = MN ? T + 4 : F64_BK + 4;
  static constexpr int SIZE = MN ? F64_BK * PITCH : T * PITCH;
  template <int V>
  __device__ static void load(double *s, const double *g, long long ld, long long mn0, long long mn, long long k0, long long k) {
    constexpr int ROWS = MN ? F64_BK : T, PER_ROW = (MN ? T : F64_BK) / V;
    const long long r0 = MN ? k0 : mn0, rows = MN ? k : mn, c0 = MN ? mn0 : k0, cols = MN ? mn : k;
#pragma unroll
    for (int i = threadIdx.x; i < ROWS * PER_ROW; i += F64_THREADS) {
      const int r = i / PER_ROW, c = (i % PER_ROW) * V;
      const long long left = r0 + r < rows ? cols - (c0 + c) : 0;
      const int valid = left >= V ? V : (left > 0 ? (int)left : 0);
      cp_async_f64<V>(s + r * PITCH + c, valid ? g + (r0 + r) * ld + c0 + c : g, valid);
    }
  }
  __device__ static double at(const double *s, int mn, int k) { return MN ? s[k * PITCH + mn] : s[mn * PITCH + k]; }
};

template <int T, bool A_MN, bool B_MN, int V>
__global__ void __launch_bounds__(F64_THREADS) gemm_f64_kernel(const __grid_constant__ GemmF64Params p) {
  ptx::grid_begin();
  using SA = SlabF64<T, A_MN>;
  using SB = SlabF64<T, B_MN>;
  constexpr int F = T / 16;  // 8 x 8 fragments of a warp along either side: its quarter of the tile is T/2 x T/2
  extern __shared__ __align__(16) double f64_smem[];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = lane >> 2, quad = lane & 3;
  const int wm = (warp >> 1) * (T / 2), wn = (warp & 1) * (T / 2);
  const int tile = blockIdx.x, split = blockIdx.y;
  const long long m0 = (long long)(tile / p.tiles_n) * T, n0 = (long long)(tile % p.tiles_n) * T;
  const double *A = p.A + (long long)blockIdx.z * p.strideA, *B = p.B + (long long)blockIdx.z * p.strideB;
  double *C = p.C + (long long)blockIdx.z * p.strideC;
  const long long slabs = (p.K + F64_BK - 1) / F64_BK;
  const long long s0 = slabs * split / p.splits, s1 = slabs * (split + 1) / p.splits;

  auto stage = [&](long long s) { return f64_smem + (int)((s - s0) % F64_STAGES) * (SA::SIZE + SB::SIZE); };
  auto queue = [&](long long s) {
    if (s < s1) {
      double *st = stage(s);
      SA::template load<V>(st, A, p.lda, m0, p.M, s * F64_BK, p.K);
      SB::template load<V>(st + SA::SIZE, B, p.ldb, n0, p.N, s * F64_BK, p.K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  double acc[F][F][2];
#pragma unroll
  for (int i = 0; i < F; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
  for (int s = 0; s < F64_STAGES - 1; ++s) queue(s0 + s);
  for (long long s = s0; s < s1; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(F64_STAGES - 2) : "memory");
    __syncthreads();  // slab s has arrived for everybody, and slab s - 1 is no longer read
    queue(s + F64_STAGES - 1);
    const double *sa = stage(s), *sb = sa + SA::SIZE;
#pragma unroll
    for (int k = 0; k < F64_BK; k += 4) {
      double a[F], b[F];
#pragma unroll
      for (int i = 0; i < F; ++i) a[i] = SA::at(sa, wm + i * 8 + row, k + quad);
#pragma unroll
      for (int j = 0; j < F; ++j) b[j] = SB::at(sb, wn + j * 8 + row, k + quad);
#pragma unroll
      for (int i = 0; i < F; ++i)
#pragma unroll
        for (int j = 0; j < F; ++j) mma_f64(acc[i][j], a[i], b[j]);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  if (p.splits > 1) {
    constexpr int PART = T * T;
    const long long t = (long long)blockIdx.z * gridDim.x + tile;
    double *part = p.ws + (t * p.splits) * PART + threadIdx.x;
#pragma unroll
    for (int i = 0; i < F; ++i)
#pragma unroll
      for (int j = 0; j < F; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) __stcg(part + split * PART + ((i * F + j) * 2 + h) * F64_THREADS, acc[i][j][h]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      s_last = atomicAdd(p.tile_count + t, 1) == p.splits - 1;
      if (s_last) p.tile_count[t] = 0;  // zero again for the next launch
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int i = 0; i < F; ++i)
#pragma unroll
      for (int j = 0; j < F; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    for (int q = 0; q < p.splits; ++q)
#pragma unroll
      for (int i = 0; i < F; ++i)
#pragma unroll
        for (int j = 0; j < F; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            acc[i][j][h] = __dadd_rn(acc[i][j][h], __ldcg(part + q * PART + ((i * F + j) * 2 + h) * F64_THREADS));
  }
#pragma unroll
  for (int i = 0; i < F; ++i) {
    const long long m = m0 + wm + i * 8 + row;
    if (m >= p.M) continue;
#pragma unroll
    for (int j = 0; j < F; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long n = n0 + wn + j * 8 + quad * 2 + h;
        if (n >= p.N) continue;
        const double o = apply_epilogue<double>(acc[i][j][h], p.ep, m, n);
        double *c = C + m * p.ldc + n;
        *c = p.ep.accumulate ? __dadd_rn(*c, o) : o;  // Incr mode: C += result
      }
  }
}

template <int T, bool A_MN, bool B_MN, int V>
static int launch_f64(b200_engine *e, const GemmF64Params &p, dim3 grid) {
  auto kern = gemm_f64_kernel<T, A_MN, B_MN, V>;
  constexpr size_t smem = sizeof(double) * F64_STAGES * (SlabF64<T, A_MN>::SIZE + SlabF64<T, B_MN>::SIZE);
  static std::atomic<int> attr_dev_mask{0};  // devices on which the attribute is set; engines on other threads share it
  if (!(attr_dev_mask & (1 << (e->device & 31)))) {
    B200_CHECK_CUDA(e, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_dev_mask |= 1 << (e->device & 31);
  }
  launch_kernel(e, kern, grid, F64_THREADS, smem, p);
  B200_CHECK_LAUNCH(e, "gemm_f64_kernel");
  return B200_OK;
}
template <int T, int V>
static int launch_f64_layout(b200_engine *e, bool a_mn, bool b_mn, const GemmF64Params &p, dim3 grid) {
  if (!a_mn && !b_mn) return launch_f64<T, false, false, V>(e, p, grid);
  if (!a_mn && b_mn) return launch_f64<T, false, true, V>(e, p, grid);
  if (a_mn && !b_mn) return launch_f64<T, true, false, V>(e, p, grid);
  return launch_f64<T, true, true, V>(e, p, grid);
}

// K may be 0: every result is then the epilogue of an empty sum.
int gemm_f64(b200_engine *e, int transA, int transB, long long M, long long N, long long K, const double *A,
             long long lda, const double *B, long long ldb, double *C, long long ldc, long long batch,
             long long strideA, long long strideB, long long strideC, const Epilogue &ep) {
  GemmF64Params p;
  p.M = M; p.N = N; p.K = K;
  p.A = A; p.B = B; p.C = C;
  p.lda = lda; p.ldb = ldb; p.ldc = ldc;
  p.strideA = strideA; p.strideB = strideB; p.strideC = strideC;
  p.ws = nullptr;
  p.tile_count = nullptr;
  p.ep = ep;
  auto tiles_of = [&](int t) { return ((M + t - 1) / t) * ((N + t - 1) / t); };
  // A 32 x 32 tile reads twice the operand bytes of a 64 x 64 one per multiply-add; it is taken only where
  // the wide tiles would leave SMs idle
  const int T = tiles_of(64) * batch >= e->sm_count ? 64 : 32;
  const long long tiles = tiles_of(T), slabs = (K + F64_BK - 1) / F64_BK;
  p.tiles_n = (int)((N + T - 1) / T);
  if (tiles >= (1LL << 31) || batch > 65535)
    return set_error(e, B200_ERR_UNSUPPORTED, "b200_gemm: %lld output tiles in %lld slices are more than one launch takes", tiles, batch);
  // k is cut until there are two blocks per SM, in pieces of at least 8 slabs: below that, leaving and
  // gathering the parts (T x T doubles each, about a microsecond per part) outweighs the shorter loop. The number
  // of tiles, and with it the cut, depends on M: not with B200_ENGINE_NO_STREAMK.
  long long splits = 1;
  if (tiles * batch < 2LL * e->sm_count && !(e->flags & B200_ENGINE_NO_STREAMK))
    splits = std::max<long long>(1, std::min<long long>({(2LL * e->sm_count + tiles * batch - 1) / (tiles * batch), slabs / 8, 16}));
  void *ws = nullptr;
  if (splits > 1 && b200_get(e, tiles * batch * splits * T * T * (long long)sizeof(double), &ws) != B200_OK)
    splits = 1;  // no room for the parts: whole k ranges
  p.splits = (int)splits;
  p.ws = (double *)ws;
  p.tile_count = e->sk_counters;  // splits > 1 only with fewer tiles than counters
  const bool vec = lda % 2 == 0 && ldb % 2 == 0 && strideA % 2 == 0 && strideB % 2 == 0 && ((uintptr_t)A | (uintptr_t)B) % 16 == 0;
  const dim3 grid((unsigned)tiles, (unsigned)splits, (unsigned)batch);
  const bool a_mn = transA != 0, b_mn = transB == 0;
  int rc;
  if (T == 64)
    rc = vec ? launch_f64_layout<64, 2>(e, a_mn, b_mn, p, grid) : launch_f64_layout<64, 1>(e, a_mn, b_mn, p, grid);
  else
    rc = vec ? launch_f64_layout<32, 2>(e, a_mn, b_mn, p, grid) : launch_f64_layout<32, 1>(e, a_mn, b_mn, p, grid);
  if (ws) b200_put(e, ws, 0);  // stream order: whoever gets the block next runs after this kernel
  return rc;
}

}  // namespace b200
