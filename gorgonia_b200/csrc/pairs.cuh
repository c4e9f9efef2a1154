// Convolutions on pairs of fp16: what a kernel reads about its operands, and how an epilogue writes the
// pairs that the next convolution reads. The arithmetic of a pair, and when pairs are usable, is in split.cu.
//
// An activation tensor in pairs form is its heads, channels innermost (NHWC), followed by its tails; its
// F16Rec lies elsewhere. A producer cannot know the largest result before it has made it, so it scales by a
// bound: largest input x largest sum of magnitudes of a filter + largest bias. For sums of a few thousand
// products that is 2^6 to 2^8 above what occurs, which leaves results down to 2^-21 of the largest with full
// pairs. The largest result that did occur is recorded for the next link's bound.
//
// Small values (split.cu) beside an ordinary one at the same place of an image are harmless: the sums they enter
// hold that one too, and they came about by cancellation, with an error above what the pair adds. A place where
// every channel is small is a place whose inputs are, and would be the whole of what some outputs of the next link
// are made from, so one such place marks the tensor. Epilogues look at the sums in front of the activation
// (Rectify leaves zeros that say nothing), in the eight or more channels that a thread has at a place, and "ordinary"
// keeps 2^7 from where pairs stop being full (kOrdinary): what 2^14 small values beside one ordinary one can add up to
// is then below that one's own rounding, so it does not matter how many small ones a tensor holds. (With at most
// n / 65536 of them, as a matrix may hold, tiny-YOLO came to 94 % of the allowance at two images and went over it at
// one, and smaller slopes leave more of them in proportion.) pairs_small_limit only keeps tensors away that consist of
// them.
#pragma once
#include "epilogue.cuh"
#include "split.h"

namespace b200 {

// In front of a constant's filters in pairs form.
struct F16Filters {
  F16Rec rec;
  unsigned l1;  // bits of the largest sum of magnitudes over a filter's taps
};

struct PairsIn {
  const F16Rec *x = nullptr;
  const F16Filters *w = nullptr;
  unsigned limit_x = 0, limit_w = 0;
};
struct PairsOut {
  __half *h = nullptr, *l = nullptr;
  F16Rec *rec = nullptr;  // null: nobody asks about the output
};

inline unsigned pairs_small_limit(long long n) { return (unsigned)(n >> 4 > 0x7FFFFFFF ? 0x7FFFFFFF : n >> 4); }

#ifdef __CUDACC__
constexpr float kOrdinary = 0.0078125f;  // 2^-7, of values scaled into fp16's range
// Kernels of the TF32 way that stand behind one of fp16 pairs run only if that turned out unusable.
__device__ __forceinline__ bool skip_launch(const int *only_if) { return only_if && __ldg(only_if) == 0; }

// Whether the operands can be used; if not, the output is marked as well, so that whoever reads it knows.
__device__ __forceinline__ bool pairs_usable(const PairsIn &in, F16Rec *out) {
  if (!f16_unusable(in.x, in.limit_x) && !f16_unusable(&in.w->rec, in.limit_w)) return true;
  if (out && blockIdx.x == 0 && threadIdx.x == 0) out->bad = 1;
  return false;
}

// Exponent that an output is scaled by (see the file comment). Called by whole warps, which share out the
// K biases.
__device__ __forceinline__ int pairs_out_exp(float amax_x, float l1, const float *bias, int K, int act, float alpha) {
  float b = 0.f;
  if (bias)
    for (int k = threadIdx.x & 31; k < K; k += 32) b = fmaxf(b, fabsf(__ldg(bias + k)));
  b = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(b)));
  float bound = amax_x * l1 * 1.0001f + b;
  if (act == B200_ACT_LEAKY) bound *= fmaxf(1.f, fabsf(alpha));
  // an infinite bound (or a NaN) takes the smallest scale: what overflows it is marked when it is stored
  const unsigned bits = bound <= 3.402823466e+38f ? __float_as_uint(bound) : 0x7F7FFFFFu;
  return f16_scale_exp(bits);
}

// What a thread has seen of an output.
struct PairStats {
  unsigned amax = 0, small = 0, bad = 0;
  __device__ __forceinline__ void see(float v) {
    const unsigned m = __float_as_uint(v) & 0x7FFFFFFFu;
    amax = amax > m ? amax : m;
  }
  // by whole warps, once
  __device__ __forceinline__ void deliver(F16Rec *rec) {
    const unsigned a = __reduce_max_sync(0xffffffffu, amax), s = __reduce_add_sync(0xffffffffu, small);
    const unsigned b = __reduce_or_sync(0xffffffffu, bad | (amax >= 0x7F800000u ? 1u : 0u));
    if ((threadIdx.x & 31) == 0) {
      // most warps have nothing larger to add: 38,000 atomic operations on one word took a pool 50 us
      if (a > *(volatile const unsigned *)&rec->amax) atomicMax(&rec->amax, a);
      if (s) atomicAdd(&rec->small, s);
      if (b) atomicOr(&rec->bad, 1u);
    }
  }
};

// N values (a multiple of 8) of one place to N / 8 16-byte pieces of heads and tails; `valid` is a multiple of 8.
// sums: the largest magnitude of the sums in front of Rectify; negative if the values themselves tell. Looked at only
// where some value is small.
template <int N>
__device__ __forceinline__ void store_pairs(const float *v, int valid, float scale, __half *h, __half *l,
                                            PairStats &st, float sums) {
  const unsigned before = st.small;
#pragma unroll
  for (int j0 = 0; j0 < N; j0 += 8) {
    if (j0 < valid) {
      __align__(16) __half hh[8], ll[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        st.small += f16_pair(v[j0 + j], scale, hh[j], ll[j]) ? 1u : 0u;
        if (!(fabsf(v[j0 + j] * scale) <= 65504.f)) st.bad = 1;
      }
      *reinterpret_cast<uint4 *>(h + j0) = *reinterpret_cast<const uint4 *>(hh);
      *reinterpret_cast<uint4 *>(l + j0) = *reinterpret_cast<const uint4 *>(ll);
    }
  }
  if (st.small != before) {
    if (sums < 0.f) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (j < valid) sums = fmaxf(sums, fabsf(v[j]));
    }
    if (sums * scale < kOrdinary) st.bad = 1;
  }
}

// What an activation leaves at least of a magnitude, unless it leaves nothing.
__device__ __forceinline__ float act_floor(int act, float alpha) {
  return act == B200_ACT_LEAKY && alpha != 0.f ? fminf(1.f, fabsf(alpha)) : 1.f;
}
// acc -> act(acc + bias), the activation chosen outside the loop. Returns what store_pairs wants to know of the sums
// in front of it: of an activation that leaves zeros, the largest magnitude. (Found for every activation it took 25 us
// of tiny-YOLO's 1690 at 64 images.)
template <int N>
__device__ __forceinline__ float finish_channels(float (&acc)[N], const float *bias, int act, float alpha) {
  if (bias) {
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = __fadd_rn(acc[j], bias[j]);
  }
  float largest = -1.f;
  if (act == B200_ACT_RECTIFY || (act == B200_ACT_LEAKY && alpha == 0.f)) {
#pragma unroll
    for (int j = 0; j < N; ++j) largest = fmaxf(largest, fabsf(acc[j]));
  }
  if (act == B200_ACT_RECTIFY) {
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = apply_act<float>(acc[j], B200_ACT_RECTIFY, alpha);
  } else if (act == B200_ACT_LEAKY) {
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = apply_act<float>(acc[j], B200_ACT_LEAKY, alpha);
  }
  return largest;
}
#endif

}  // namespace b200
