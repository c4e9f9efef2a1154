// Splitting float32 operands into pairs of narrower values for the tensor cores (split.cu).
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "tc_operand.h"

struct b200_engine;

namespace b200 {

// What is known about a tensor that was split into pairs of fp16 (see split.cu): written by the kernels
// that make the pairs, read by those that multiply them.
struct F16Rec {
  unsigned amax;   // bits of the largest magnitude among the finite values
  unsigned small;  // values that are too small for a full pair (nonzero, below 2^-14 after scaling)
  unsigned bad;    // nonzero: an infinity or NaN is among the values, or a line of small values (split.cu)
  int scale_exp;   // the values were scaled by 2^scale_exp
};
// A tensor of n values may hold this many that are too small for a full pair.
__host__ __device__ inline unsigned f16_small_limit(long long n) {
  return (unsigned)(n >> 16 > 0x7FFFFFFF ? 0x7FFFFFFF : n >> 16);
}

// One operand as it lies in memory and where its pairs go: rows padded to `ldo` values with zeros.
struct SplitJob {
  const float *src = nullptr;
  long long ld = 0, stride = 0, rows = 0, cols = 0, batch = 0;
  void *hi = nullptr, *lo = nullptr;
  long long ldo = 0;
  // fp16 pairs only: the record, how many small values it allows, and along what they are summed
  F16Rec *rec = nullptr;
  unsigned limit = 0;
  unsigned lines = 0;  // kLineRows and / or kLineCols
};
constexpr unsigned kLineRows = 1, kLineCols = 2;

// Each takes one or two operands in one launch (b.src == null: one).
int launch_split_tf32(b200_engine *e, const SplitJob &a, const SplitJob &b);
// The pairs of fp16: the largest magnitude first, then the split. rec must be zero before.
int launch_split_f16(b200_engine *e, const SplitJob &a, const SplitJob &b);
// The TF32 split for the case that the fp16 pairs of a product turned out unusable: runs only if one of the
// two records says so, and leaves that answer in *redo for the product that follows.
int launch_split_tf32_redo(b200_engine *e, const SplitJob &a, const SplitJob &b, const F16Rec *ra, unsigned limit_a,
                           const F16Rec *rb, unsigned limit_b, int *redo);

// The largest magnitude of n values, or of a sample of them (step > 1), into rec.
int launch_magnitude(b200_engine *e, const float *x, long long n, int step, F16Rec *rec);
// Whether any of k <= kMaxPairsRecs records, one after the other in memory, says that its tensor is unusable
// goes to *verdict; the records are cleared.
constexpr int kMaxPairsRecs = 32;
// The engine's own records are zero between calls: a call that gave up before the launch that clears them puts
// them back with this.
void clear_f16_recs(b200_engine *e);
int launch_pairs_check(b200_engine *e, F16Rec *recs, const unsigned *limits, int k, int *verdict);

#ifdef __CUDACC__
// Scale that brings a largest magnitude (bits of a finite float >= 0) into [2^14, 2^15): at least 2^-113.
// Kept below 2^110 so that it and its inverse are normal numbers; values that this leaves small are counted.
__device__ __forceinline__ int f16_scale_exp(unsigned amax_bits) {
  const int e = 14 - ((int)(amax_bits >> 23) - 127);
  return e > 110 ? 110 : e;
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((unsigned)(127 + e) << 23); }  // |e| <= 126
// The factors that take a product of scaled operands back: two, so that neither is out of range and no
// intermediate result overflows where the final one does not.
__device__ __forceinline__ void f16_unscale(int exp_a, int exp_b, float &s1, float &s2) {
  const int t = -(exp_a + exp_b), t1 = t < -126 ? -126 : (t > 126 ? 126 : t);
  s1 = pow2(t1);
  s2 = pow2(t - t1);
}
__device__ __forceinline__ bool f16_unusable(const F16Rec *r, unsigned limit) {
  return *(volatile const unsigned *)&r->bad != 0 || *(volatile const unsigned *)&r->small > limit;
}
constexpr float kFullPair = 6.103515625e-05f;  // 2^-14, fp16's smallest normal number
// x * 2^e -> head and tail; true if the value is too small for a full pair
__device__ __forceinline__ bool f16_pair(float x, float scale, __half &h, __half &l) {
  const float xs = x * scale;
  h = __float2half_rn(xs);
  l = __float2half_rn((xs - __half2float(h)) * 2048.f);
  return x != 0.f && fabsf(xs) < kFullPair;
}
// n small values more. Whether it is still worth looking what they lie among: not once the record says that
// the tensor is unusable.
__device__ __forceinline__ bool f16_count_small(F16Rec *r, unsigned limit, unsigned n) {
  if (f16_unusable(r, limit)) return false;
  return atomicAdd(&r->small, n) + n <= limit;
}
#endif

}  // namespace b200
