// float32 operands as pairs of narrower values whose products the tensor cores add up in float32.
//
// TF32 pairs: x = head + tail, both TF32 (11 significant bits) in float32 containers, 8 bytes per value.
//
// fp16 pairs: the whole operand is scaled by the power of two that brings its largest magnitude into
// [2^14, 2^15); then x * 2^e = head + tail * 2^-11 with head = fp16(x * 2^e) and tail = fp16 of the (exact)
// remainder times 2^11. fp16 has the 11 significant bits of TF32, so the pair carries x as closely as the
// TF32 pair does, in half the bytes and at twice the tensor-core rate. What fp16 lacks is range: a small
// value, below 2^-14 after scaling (2^-29 of the largest), keeps an absolute error of 2^-36 instead of a
// relative one. Beside a value of the full range in the same sum that is no more than that one's rounding
// (2^-22 of at least 2^-14); where every value along k is small, a whole row or column of the product would
// lose its bits. Small values are therefore counted in the operand's F16Rec, which also notes infinities and
// NaNs, and each of them looks for a value of full range in its line along k. A product whose operands hold
// more than n / 65536 small values, one that is alone, an infinity or a NaN, is made from TF32 pairs instead:
// the kernels of both ways are launched, and one of them returns at once (the host never waits to find out).
// N(0, 1) draws hold about one small value in 10^8, and its neighbour is an ordinary one: looking costs nothing.
//
// All of these passes are bound by HBM: 4 bytes read and 4 (fp16) or 8 (TF32) written per value. A thread
// takes eight (four) neighbouring columns, 16 bytes per store; both operands of a product share a launch.
// The row-wise and element-wise kernels this replaces took a launch per operand, and 7 to 10 us for 2.5 MB
// with a pitch that is no multiple of four, most of it 64-bit divisions.
#include "split.h"

#include <algorithm>

#include "engine.h"
#include "ptx.cuh"

namespace b200 {

enum { SPLIT_AMAX, SPLIT_F16, SPLIT_TF32, SPLIT_TF32_REDO };

struct SplitRedo {
  const F16Rec *ra, *rb;
  unsigned limit_a, limit_b;
  int *redo;
};

__device__ __forceinline__ float split_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// Whether the line through element (row, col) of a slice holds a value of full range among the kLineReach
// nearest after it (the line taken as a ring). By a whole warp.
constexpr int kLineReach = 4096;
__device__ bool line_has_full(const float *first, long long step, long long len, long long at, float scale) {
  const int lane = threadIdx.x & 31;
  const long long reach = len < kLineReach ? len : kLineReach;
  for (long long o = 0; o < reach; o += 128) {
    bool full = false;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long d = o + q * 32 + lane;
      if (d < reach) {
        const long long i = at + d < len ? at + d : at + d - len;
        full |= fabsf(__ldg(first + i * step)) * scale >= kFullPair;
      }
    }
    if (__any_sync(0xffffffffu, full)) return true;
  }
  return false;
}

// The rare end of SPLIT_F16's step: `mine` marks the small ones of this lane's eight values, which begin at
// column c0 of row r of the slice at `slice`. By a whole warp. Returns whether the operand is known to be of no use, so
// that the warp need not ask again.
__device__ __noinline__ bool note_small(const SplitJob &j, unsigned mine, const float *slice, long long r, long long c0,
                                        float scale) {
  const int lane = threadIdx.x & 31;
  const unsigned n = __reduce_add_sync(0xffffffffu, (unsigned)__popc(mine));
  bool look = false;
  if (lane == 0) look = f16_count_small(j.rec, j.limit, n);
  if (!__shfl_sync(0xffffffffu, look, 0)) return true;
  for (unsigned lanes = __ballot_sync(0xffffffffu, mine != 0); lanes; lanes &= lanes - 1) {
    const int src = __ffs(lanes) - 1;
    const long long lr = __shfl_sync(0xffffffffu, r, src), lc0 = __shfl_sync(0xffffffffu, c0, src);
    const float *ls = (const float *)__shfl_sync(0xffffffffu, (unsigned long long)slice, src);
    for (unsigned m = __shfl_sync(0xffffffffu, mine, src); m; m &= m - 1) {
      // others may have found out meanwhile: one warp that went on through 256 values took 470 us
      if (__shfl_sync(0xffffffffu, (int)f16_unusable(j.rec, j.limit), 0)) return true;
      const long long lc = lc0 + __ffs(m) - 1;
      bool alone = false;
      if (j.lines & kLineRows) alone = !line_has_full(ls + lr * j.ld, 1, j.cols, lc, scale);
      if (!alone && (j.lines & kLineCols)) alone = !line_has_full(ls + lc, j.ld, j.rows, lr, scale);
      if (alone) {
        if (lane == 0) atomicOr(&j.rec->bad, 1u);
        return true;
      }
    }
  }
  return false;
}

template <int MODE>
__global__ void __launch_bounds__(256) split_kernel(const __grid_constant__ SplitJob ja, const __grid_constant__ SplitJob jb,
                                                    int blocks_a, SplitRedo redo) {
  ptx::grid_begin();
  constexpr int V = MODE == SPLIT_TF32 || MODE == SPLIT_TF32_REDO ? 4 : 8;
  __shared__ unsigned s_red[8], s_bad[8];
  if (MODE == SPLIT_TF32_REDO) {
    // one thread asks for its block: a million threads reading the same words took 41 us
    if (threadIdx.x == 0) {
      s_bad[0] = f16_unusable(redo.ra, redo.limit_a) || f16_unusable(redo.rb, redo.limit_b) ? 1u : 0u;
      if (blockIdx.x == 0) *redo.redo = (int)s_bad[0];
    }
    __syncthreads();
    if (s_bad[0] == 0) return;
  }
  const bool second = (int)blockIdx.x >= blocks_a;
  const SplitJob &j = second ? jb : ja;
  const float *src = j.src;
  const long long ld = j.ld, stride = j.stride, rows = j.rows, cols = j.cols;
  const long long per_row = (MODE == SPLIT_AMAX ? (cols + V - 1) / V : j.ldo / V);
  const long long total = rows * j.batch * per_row;
  const bool vec = ((ld | stride) & 3) == 0 && ((uintptr_t)src & 15) == 0;
  const int nblk = second ? (int)gridDim.x - blocks_a : blocks_a, blk = second ? (int)blockIdx.x - blocks_a : (int)blockIdx.x;
  const bool narrow = total <= 0xFFFFFFFFLL;  // 32-bit divisions
  float scale = 0.f;
  if (MODE == SPLIT_F16) {
    const int ex = f16_scale_exp(*(volatile const unsigned *)&j.rec->amax);
    scale = pow2(ex);
    if (blk == 0 && threadIdx.x == 0) j.rec->scale_exp = ex;
  }
  unsigned amax = 0, bad = 0;
  bool useless = false;  // SPLIT_F16: the record has been seen to say so
  // SPLIT_F16: warps stay whole for note_small
  const long long lane_off = MODE == SPLIT_F16 ? threadIdx.x & 31 : 0;
  for (long long t = (long long)blk * 256 + threadIdx.x; t - lane_off < total; t += (long long)nblk * 256) {
    unsigned small = 0;
    const float *slice = nullptr;
    long long r = 0, c0 = 0;
    if (MODE != SPLIT_F16 || t < total) {
      long long row, g, b;
      if (narrow) {
        const uint32_t rr = (uint32_t)t / (uint32_t)per_row, bb = rr / (uint32_t)rows;
        row = rr;
        g = (uint32_t)t - rr * (uint32_t)per_row;
        b = bb;
        r = rr - bb * (uint32_t)rows;
      } else {
        row = t / per_row;
        g = t - row * per_row;
        b = row / rows;
        r = row - b * rows;
      }
      c0 = g * V;
      slice = src + b * stride;
      const float *p = slice + r * ld + c0;
      float x[V];
      if (vec && c0 + V <= cols) {
#pragma unroll
        for (int q = 0; q < V / 4; ++q) {
          const float4 v = __ldg(reinterpret_cast<const float4 *>(p) + q);
          x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q) x[q] = c0 + q < cols ? __ldg(p + q) : 0.f;
      }
      if (MODE == SPLIT_AMAX) {
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const unsigned m = __float_as_uint(x[q]) & 0x7FFFFFFFu;
          if (m >= 0x7F800000u) bad = 1;
          else amax = amax > m ? amax : m;
        }
      } else if (MODE == SPLIT_F16) {
        __align__(16) __half h[V], l[V];
#pragma unroll
        for (int q = 0; q < V; ++q) small |= f16_pair(x[q], scale, h[q], l[q]) ? 1u << q : 0u;
        reinterpret_cast<uint4 *>(j.hi)[t] = *reinterpret_cast<const uint4 *>(h);
        reinterpret_cast<uint4 *>(j.lo)[t] = *reinterpret_cast<const uint4 *>(l);
      } else {
        float h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          h[q] = split_tf32(x[q]);
          l[q] = split_tf32(__fsub_rn(x[q], h[q]));
        }
        reinterpret_cast<float4 *>(j.hi)[t] = make_float4(h[0], h[1], h[2], h[3]);
        reinterpret_cast<float4 *>(j.lo)[t] = make_float4(l[0], l[1], l[2], l[3]);
      }
    }
    if (MODE == SPLIT_F16 && !useless && __any_sync(0xffffffffu, small != 0))
      useless = note_small(j, small, slice, r, c0, scale);
  }
  if (MODE == SPLIT_AMAX) {
    amax = __reduce_max_sync(0xffffffffu, amax);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
      s_red[threadIdx.x >> 5] = amax;
      s_bad[threadIdx.x >> 5] = bad;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w) {
        amax = amax > s_red[w] ? amax : s_red[w];
        bad |= s_bad[w];
      }
      atomicMax(&j.rec->amax, amax);
      if (bad) atomicOr(&j.rec->bad, 1u);
    }
  }
}

template <int MODE>
static int launch_split(b200_engine *e, const SplitJob &a, const SplitJob &b, const SplitRedo &redo) {
  constexpr int V = MODE == SPLIT_TF32 || MODE == SPLIT_TF32_REDO ? 4 : 8;
  auto blocks_of = [&](const SplitJob &j) -> long long {
    if (!j.src) return 0;
    const long long groups = j.rows * j.batch * ((j.cols + V - 1) / V);
    // the launch that usually finds nothing to do has no more blocks than start at once
    const long long most = MODE == SPLIT_TF32_REDO ? e->sm_count * 4LL : e->sm_count * 16LL;
    return std::max<long long>(1, std::min<long long>((groups + 255) / 256, most));
  };
  const long long ba = blocks_of(a), bb = blocks_of(b);
  if (ba + bb == 0) return B200_OK;
  launch_kernel(e, split_kernel<MODE>, (int)(ba + bb), 256, 0, a, b, (int)ba, redo);
  B200_CHECK_LAUNCH(e, "split_kernel");
  return B200_OK;
}

int launch_split_tf32(b200_engine *e, const SplitJob &a, const SplitJob &b) {
  return launch_split<SPLIT_TF32>(e, a, b, SplitRedo());
}
int launch_split_f16(b200_engine *e, const SplitJob &a, const SplitJob &b) {
  const int rc = launch_split<SPLIT_AMAX>(e, a, b, SplitRedo());
  return rc != B200_OK ? rc : launch_split<SPLIT_F16>(e, a, b, SplitRedo());
}
int launch_split_tf32_redo(b200_engine *e, const SplitJob &a, const SplitJob &b, const F16Rec *ra, unsigned limit_a,
                           const F16Rec *rb, unsigned limit_b, int *redo) {
  return launch_split<SPLIT_TF32_REDO>(e, a, b, SplitRedo{ra, rb, limit_a, limit_b, redo});
}

// The largest magnitude of n values into rec->amax, and rec->bad for infinities and NaNs; with step > 1, of
// every step-th 4 KB only where there are more than 4 MB.
__global__ void __launch_bounds__(256) magnitude_kernel(const float *__restrict__ x, long long n, int step, F16Rec *rec) {
  ptx::grid_begin();
  __shared__ unsigned s_max[8], s_bad[8];
  unsigned amax = 0, bad = 0;
  auto see = [&](float v) {
    const unsigned m = __float_as_uint(v) & 0x7FFFFFFFu;
    if (m >= 0x7F800000u) bad = 1;
    else amax = amax > m ? amax : m;
  };
  const long long groups = (n + 1023) / 1024;
  if (n <= (1 << 20)) step = 1;
  const bool vec = ((uintptr_t)x & 15) == 0;
  for (long long g = (long long)blockIdx.x * step; g < groups; g += (long long)gridDim.x * step) {
    const long long i = g * 1024 + threadIdx.x * 4;
    if (vec && i + 4 <= n) {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(x + i));
      see(v.x); see(v.y); see(v.z); see(v.w);
    } else {
      for (long long k = i; k < i + 4 && k < n; ++k) see(__ldg(x + k));
    }
  }
  amax = __reduce_max_sync(0xffffffffu, amax);
  bad = __reduce_or_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    s_max[threadIdx.x >> 5] = amax;
    s_bad[threadIdx.x >> 5] = bad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      amax = amax > s_max[w] ? amax : s_max[w];
      bad |= s_bad[w];
    }
    if (amax) atomicMax(&rec->amax, amax);
    if (bad) atomicOr(&rec->bad, 1u);
  }
}
int launch_magnitude(b200_engine *e, const float *x, long long n, int step, F16Rec *rec) {
  const long long groups = ((n + 1023) / 1024 + (n > (1 << 20) ? step : 1) - 1) / (n > (1 << 20) ? step : 1);
  launch_kernel(e, magnitude_kernel, (int)std::max<long long>(1, std::min<long long>(groups, e->sm_count * 8LL)), 256, 0, x, n, step, rec);
  B200_CHECK_LAUNCH(e, "magnitude_kernel");
  return B200_OK;
}

// Whether any of k records says that its tensor is unusable; clears them for the next round.
struct PairsLimits {
  unsigned limit[kMaxPairsRecs];
};
__global__ void pairs_check_kernel(F16Rec *recs, PairsLimits l, int k, int *verdict) {
  ptx::grid_begin();
  const int i = threadIdx.x;
  const bool bad = i < k && f16_unusable(recs + i, l.limit[i]);
  const bool any = __any_sync(0xffffffffu, bad);
  if (i < k) recs[i] = F16Rec{0, 0, 0, 0};
  if (i == 0) *verdict = any ? 1 : 0;
}
int launch_pairs_check(b200_engine *e, F16Rec *recs, const unsigned *limits, int k, int *verdict) {
  PairsLimits l;
  for (int i = 0; i < kMaxPairsRecs; ++i) l.limit[i] = i < k ? limits[i] : 0xFFFFFFFFu;
  launch_kernel(e, pairs_check_kernel, 1, 32, 0, recs, l, k, verdict);
  B200_CHECK_LAUNCH(e, "pairs_check_kernel");
  return B200_OK;
}
void clear_f16_recs(b200_engine *e) {
  if (cudaMemsetAsync(e->f16_recs, 0, 256, e->stream) != cudaSuccess) cudaGetLastError();  // the call's own error is told
}

}  // namespace b200
