// Matrix multiply on the 5th-generation tensor cores (tcgen05), operands fed by TMA, accumulators
// in tensor memory. Stands where Engine.MatMul calls cuBLAS Sgemm in gorgonia
// (cuda/linalg.go:110-229) and where batchedMatMul loops over slices (operatorLinAlg.go:435-502).
//
// One persistent CTA per SM, 10 warps with fixed roles:
//   warp 0     TMA producer: one lane queues the A and B boxes of each k-block into a ring of
//              shared-memory stages (128-byte swizzle) and arms the stage's "full" mbarrier;
//   warp 1     MMA issuer: one lane issues tcgen05.mma for each 32-byte k-slice of a stage,
//              commits the stage's "empty" mbarrier when the tensor core has read it, and commits
//              the accumulator's "full" mbarrier after the last k-block. Owns the TMEM allocation;
//   warps 2-9  epilogue: each drains one half of the columns of its 32-lane quarter of the
//              accumulator with tcgen05.ld, applies the fused bias/activation and stores rows of C
//              with 128-bit stores.
// The accumulator is double-buffered in TMEM (2 x BN columns), so the epilogue of tile i runs
// while the MMAs of tile i+1 are issued.
//
// Operand layouts. tcgen05 takes either operand K-major (k contiguous in memory) or MN-major
// (m resp. n contiguous). Row-major A (M x K) is K-major, row-major B (K x N) is MN-major; the
// transposed storages swap that. All four combinations run without a transposing pass: only the
// TMA box shape and two fields of the shared-memory descriptor differ.
//
// float32 runs on pairs of narrower values (split.cu): each operand is split once into heads and tails
// (x = hi + lo up to 2^-22 relative), and the products hi*hi, hi*lo and lo*hi are accumulated in fp32. The
// split is a streaming pass into arena scratch; the main loop then loads four tiles per stage. Two kinds:
//   TF32 (TERMS 3): any float32 values; 32 k per 128-byte row.
//   fp16 (TERMS 2): 64 k per 128-byte row and twice the tensor rate, so half the shared-memory traffic and
//     half the tensor time for a product, with the same 11 + 11 significant bits, for operands whose values
//     lie within 2^-29 of their largest (nearly all of them: F16Rec). Operands that do not are found on the
//     device; the kernel then returns at once and the TF32 launch behind it makes the product.
//     4096^3: 591 -> 317 us alone, 642 -> 400 with all passes; 8192^3 5106 -> 2870 with all passes.
//
// CTA pairs (PAIR, bf16 only): large problems run as clusters of two CTAs on neighbouring SMs that
// share one 256-row tile: each CTA loads its own 128 rows of A and only half of the tile's B rows,
// the even CTA issues tcgen05.mma.cta_group::2 (M = 256), which reads both halves of B across the
// pair, and each CTA drains its own 128 rows of the accumulator. A CTA then brings a third less
// into shared memory per k-block. The stage's "full" barrier lives in the even CTA and counts the
// bytes of both CTAs' loads; "empty" and "accumulator full" exist in both and the even CTA's commits
// name each in turn; "accumulator empty" lives in the even CTA and takes the arrivals of both
// epilogues. 3xTF32 does not pair up: its wide instruction A_head x [B_head | B_tail] would take
// B_head from one CTA and B_tail from the other, A_tail x B_head then needs half of B_head in each
// at one common offset, i.e. a second, half-size slab, and with 7/8 of the bytes per CTA the pair
// measured no faster than two CTAs on their own.
//
// No TMA multicast anywhere: every CTA loads its own tiles from local HBM.
// Every mbarrier wait is bounded; a wait that runs out raises the engine's error word and all
// roles leave their loops, TMEM is released and the kernel returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "engine.h"
#include "epilogue.cuh"
#include "ptx.cuh"
#include "split.h"
#include "tc_common.cuh"
#include "tc_operand.h"

namespace b200 {

int gemm_simt(b200_engine *e, int dtype, int transA, int transB, long long M, long long N, long long K,
              const void *A, long long lda, const void *B, long long ldb, void *C, long long ldc, long long batch,
              long long strideA, long long strideB, long long strideC, const Epilogue &ep);

// ------------------------------------------------------------------------------------------
// kernel
// ------------------------------------------------------------------------------------------

constexpr int TC_BM = 128;
constexpr int TC_THREADS = 320;  // 10 warps: TMA, MMA, 8 epilogue
constexpr int TC_ROW_BYTES = 128;  // one swizzle row: 64 bf16 or 32 fp32 along the contiguous dim

struct GemmTcParams {
  long long M, N, K, batch;
  void *C;                      // may be null when only the split form is wanted
  long long ldc, strideC;
  float *C_hi, *C_lo;           // C additionally as TF32 head / tail with row pitch ld_split, or null
  long long ld_split;
  int tiles_m, tiles_n, num_k;  // num_k = k-blocks of BK elements
  int chunk_k;                  // k-blocks accumulated in tensor memory before the epilogue folds them
  int group_m;                  // rasterisation: m-blocks per group
  int stages;
  int c_vec;                    // 1: rows of C can be stored with 128-bit stores
  int a_zmul, b_zmul;           // 0: the operand is shared by all batch entries (z coordinate 0)
  // how the work is shared between the CTAs (TilePieces, tc_common.cuh); 3xTF32 only
  int streamk;
  int units;                    // tiles * num_k (0 when the k range is not shared)
  float *ws;                    // partial tiles, 2 slots of TC_BM x BN floats per CTA
  int *tile_count;              // parts delivered per tile; zero between launches
  int workers;                  // CTAs, or CTA pairs, that share the tiles out
  int sk_first, sk_workers;     // k ranges are shared from this tile on, among this many CTAs (TilePieces)
  // fp16 pairs: what is known about the operands; the launch does nothing if either is unusable
  const F16Rec *rec_a, *rec_b;
  unsigned limit_a, limit_b;
  // TF32 pairs behind a launch of fp16 pairs: nothing is done unless *redo; clears the records of the
  // operands that were split for this product alone
  const int *redo;
  F16Rec *clear_a, *clear_b;
  Epilogue ep;
  int *err_flag;
};

// TERMS = 1: bf16 operands (kind::f16). TERMS = 3: fp32 as pairs of TF32 (kind::tf32), TERMS = 2: as pairs of
// fp16 (kind::f16); tensor maps 0/1 = head/tail of A, 2/3 = head/tail of B.
// PAIR: two CTAs per 256-row tile (see the file comment); then B's map has a box of BN / 2 rows.
template <int TERMS, int BN, bool A_MN, bool B_MN, bool PAIR>
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                   const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1,
                   const __grid_constant__ GemmTcParams p) {
  ptx::grid_begin();
  static_assert(!PAIR || TERMS == 1, "only bf16 tiles are shared by a pair of CTAs");
  constexpr int ES = TERMS == 3 ? 4 : 2;           // operand element size
  constexpr int BK = TC_ROW_BYTES / ES;            // k elements per stage: 64 (16-bit values) / 32 (TF32)
  constexpr int UK = 32 / ES;                      // k elements per MMA: 16 / 8
  constexpr int NSPLIT = TERMS == 1 ? 1 : 2;       // copies of each operand per stage (head, tail)
  constexpr int A_BYTES = TC_BM * TC_ROW_BYTES;    // 16 KB
  constexpr int B_BYTES = BN * TC_ROW_BYTES;
  constexpr int BH_BYTES = B_BYTES / 2;            // half of the tile's B rows
  // what one CTA holds per stage. Alone: every copy of A and B. In a pair: its A rows and its half of B
  constexpr int STAGE_BYTES = !PAIR ? NSPLIT * (A_BYTES + B_BYTES) : A_BYTES + BH_BYTES;
  constexpr int MN_PER_BOX = TC_ROW_BYTES / ES;    // m/n elements covered by one MN-major box
  constexpr int MMA_M = PAIR ? 2 * TC_BM : TC_BM;
  constexpr int FMT = TERMS == 1 ? 1 : (TERMS == 2 ? 0 : 2);  // bf16, fp16, TF32
  constexpr uint32_t IDESC = make_idesc(FMT, A_MN, B_MN, MMA_M, BN);
  // pairs: B's head and tail slabs are adjacent in shared memory, and so are the main and the
  // cross-term accumulator in tensor memory, so A_head x [B_head | B_tail] is ONE instruction of
  // width 2*BN. An instruction costs a fixed ~65 cycles on top of its arithmetic: two per k step
  // beat three.
  constexpr uint32_t IDESC_WIDE = make_idesc(FMT, A_MN, B_MN, MMA_M, TERMS == 1 ? BN : 2 * BN);
  constexpr int MAX_STAGES = 8;
  // TMEM columns of one accumulator buffer: pairs keep the cross terms in a second accumulator
  constexpr int ACC_COLS = TERMS == 1 ? BN : 2 * BN;
  constexpr int TMEM_COLS = 2 * ACC_COLS;  // double-buffered; a power of two >= 32 for every BN used

  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_full[2], acc_empty[2];
  __shared__ __align__(8) uint64_t epi_bar;  // the 8 epilogue warps meet here when a partial tile is handed over
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_fail, s_last;

  // which of the two float32 launches makes the product (the same answer in every thread of the grid)
  if (TERMS == 2 && (f16_unusable(p.rec_a, p.limit_a) || f16_unusable(p.rec_b, p.limit_b))) return;
  if (TERMS == 3 && p.redo) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      if (p.clear_a) *p.clear_a = F16Rec{0, 0, 0, 0};
      if (p.clear_b) *p.clear_b = F16Rec{0, 0, 0, 0};
    }
    if (*(volatile const int *)p.redo == 0) return;
  }
  // the ring must start on a 1024-byte boundary for the 128-byte swizzle
  unsigned char *smem = reinterpret_cast<unsigned char *>(((uintptr_t)tc_smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int stages = p.stages;
  const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;  // 0: the CTA that issues the pair's MMAs
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int tiles_per_batch = p.tiles_m * p.tiles_n;  // the host refuses launches of 2^31 tiles
  const int total_tiles = tiles_per_batch * (int)p.batch;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&acc_full[b], 1);
      ptx::mbar_init(&acc_empty[b], PAIR ? 16 : 8);  // one arrival per epilogue warp (of both CTAs)
    }
    ptx::mbar_init(&epi_bar, 8);
    ptx::fence_mbar_init();
    s_fail = 0;
    s_last = 0;
  }
  if (warp == 1) {
    if (PAIR) {
      ptx::tmem_alloc_pair(&tmem_base_s, TMEM_COLS);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(&tmem_base_s, TMEM_COLS);
      ptx::tmem_relinquish();
    }
  }
  if (warp == 0 && lane == 0) {
    ptx::prefetch_tmap(&tmA0);
    ptx::prefetch_tmap(&tmB0);
    if (TERMS != 1) {
      ptx::prefetch_tmap(&tmA1);
      ptx::prefetch_tmap(&tmB1);
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (PAIR) ptx::cluster_sync();  // the other CTA's barriers are initialised before anything reaches them
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  // shared::cluster address of a barrier of the even CTA / of the other CTA
  auto at_leader = [&](uint64_t *bar) { return PAIR ? ptx::map_to_rank(ptx::smem_addr(bar), 0u) : ptx::smem_addr(bar); };
  auto at_peer = [&](uint64_t *bar) { return ptx::map_to_rank(ptx::smem_addr(bar), rank ^ 1u); };

  // tile index -> (batch, m block, n block); m blocks are walked in groups so that the CTAs of
  // one wave share B columns and A rows in L2
  auto decode = [&](int tile, int &bz, int &mb, int &nb) {
    bz = tile / tiles_per_batch;
    const int t = tile - bz * tiles_per_batch;
    const int per_group = p.group_m * p.tiles_n;
    const int g = t / per_group;
    const int first_m = g * p.group_m;
    const int gm = (p.tiles_m - first_m) < p.group_m ? (p.tiles_m - first_m) : p.group_m;
    const int r = t % per_group;
    mb = first_m + r % gm;
    nb = r / gm;
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      TilePieces pieces(p.streamk, p.units, p.num_k, total_tiles, worker, p.workers, p.sk_first, p.sk_workers);
      int tile, kb0, kb1;
      while (ok && pieces.next(tile, kb0, kb1)) {
        int bz, mb, nb;
        decode(tile, bz, mb, nb);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
            ok = false;
            break;
          }
          unsigned char *st = smem + (size_t)stage * STAGE_BYTES;
          const int k0 = kb * BK;
          if (PAIR) {
            // the even CTA arms the stage for the bytes of both CTAs; the odd CTA's bytes may land
            // first, which only drives the pending count below zero for a moment
            if (rank == 0) ptx::mbar_arrive_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
            const uint32_t fb = at_leader(&full_bar[stage]);
            const int m0 = (mb * 2 + (int)rank) * TC_BM;
            if (!A_MN) {
              ptx::tma_load_3d_pair(st, &tmA0, k0, m0, bz * p.a_zmul, fb);
            } else {
#pragma unroll
              for (int q = 0; q < TC_BM / MN_PER_BOX; ++q)
                ptx::tma_load_3d_pair(st + q * (BK * TC_ROW_BYTES), &tmA0, m0 + q * MN_PER_BOX, k0, bz * p.a_zmul, fb);
            }
            unsigned char *sb = st + A_BYTES;
            const int nh = nb * BN + (int)rank * (BN / 2);  // this CTA's half of the tile's B rows
            if (!B_MN) {
              ptx::tma_load_3d_pair(sb, &tmB0, k0, nh, bz * p.b_zmul, fb);  // box of BN / 2 rows
            } else {
#pragma unroll
              for (int q = 0; q < BN / 2 / MN_PER_BOX; ++q)
                ptx::tma_load_3d_pair(sb + q * (BK * TC_ROW_BYTES), &tmB0, nh + q * MN_PER_BOX, k0, bz * p.b_zmul, fb);
            }
          } else {
            ptx::mbar_arrive_expect_tx(&full_bar[stage], STAGE_BYTES);
#pragma unroll
            for (int h = 0; h < NSPLIT; ++h) {
              const CUtensorMap *ta = h == 0 ? &tmA0 : &tmA1;
              const CUtensorMap *tb = h == 0 ? &tmB0 : &tmB1;
              unsigned char *sa = st + h * A_BYTES;
              unsigned char *sb = st + NSPLIT * A_BYTES + h * B_BYTES;
              if (!A_MN) {
                ptx::tma_load_3d(sa, ta, k0, mb * TC_BM, bz * p.a_zmul, &full_bar[stage]);
              } else {
#pragma unroll
                for (int q = 0; q < TC_BM / MN_PER_BOX; ++q)
                  ptx::tma_load_3d(sa + q * (BK * TC_ROW_BYTES), ta, mb * TC_BM + q * MN_PER_BOX, k0,
                                   bz * p.a_zmul, &full_bar[stage]);
              }
              if (!B_MN) {
                ptx::tma_load_3d(sb, tb, k0, nb * BN, bz * p.b_zmul, &full_bar[stage]);
              } else {
#pragma unroll
                for (int q = 0; q < BN / MN_PER_BOX; ++q)
                  ptx::tma_load_3d(sb + q * (BK * TC_ROW_BYTES), tb, nb * BN + q * MN_PER_BOX, k0,
                                   bz * p.b_zmul, &full_bar[stage]);
              }
            }
          }
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) s_fail = 1;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (of a pair: the even CTA's only) ----------------
    if (lane == 0 && rank == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int use = 0;  // accumulator-buffer uses so far (one per k-chunk)
      bool ok = true;
      // descriptors of stage 0, k-slice 0; a later stage adds its byte offset >> 4, a later k-slice
      // 32 bytes along a K-major row or UK k-rows of an MN-major block (the steps the helpers take)
      constexpr int A_STEP = (A_MN ? UK * TC_ROW_BYTES : 32) >> 4, B_STEP = (B_MN ? UK * TC_ROW_BYTES : 32) >> 4;
      const uint32_t st0 = ptx::smem_addr(smem);
      uint64_t a_desc0[NSPLIT], b_desc0[NSPLIT];
#pragma unroll
      for (int h = 0; h < NSPLIT; ++h) {
        a_desc0[h] = make_smem_desc(st0 + h * A_BYTES, A_MN ? BK * TC_ROW_BYTES : 16, (A_MN && ES == 4) ? 512 : 1024,
                                    (A_MN && ES == 4) ? 1 : 2);
        // pair: this CTA's half of B
        b_desc0[h] = make_smem_desc(st0 + NSPLIT * A_BYTES + h * B_BYTES, B_MN ? BK * TC_ROW_BYTES : 16,
                                    (B_MN && ES == 4) ? 512 : 1024, (B_MN && ES == 4) ? 1 : 2);
      }
      const uint32_t full0 = ptx::smem_addr(&full_bar[0]), empty0 = ptx::smem_addr(&empty_bar[0]);
      const uint32_t empty0_peer = PAIR ? ptx::map_to_rank(empty0, 1u) : 0u;
      uint32_t ready = 0;  // the poll behind the previous k-block saw this stage's barrier complete
      TilePieces pieces(p.streamk, p.units, p.num_k, total_tiles, worker, p.workers, p.sk_first, p.sk_workers);
      int tile, kb0, kb1;
      while (ok && pieces.next(tile, kb0, kb1)) {
        for (int kc = kb0; kc < kb1 && ok; kc += p.chunk_k, ++use) {
          const int buf = use & 1;
          const uint32_t acc_phase = (uint32_t)((use >> 1) & 1);
          // the epilogue must have drained this accumulator buffer (first use passes at once)
          if (!ptx::mbar_wait(&acc_empty[buf], acc_phase ^ 1)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t d_main = tmem_base + (uint32_t)(buf * ACC_COLS);
          const uint32_t d_tail = d_main + BN;  // pairs only: the small cross terms
          const int kend = kc + p.chunk_k < kb1 ? kc + p.chunk_k : kb1;
          for (int kb = kc; kb < kend; ++kb) {
            if (!ready && !ptx::mbar_wait(&full_bar[stage], phase)) {
              ok = false;
              break;
            }
            ptx::tc_fence_after_sync();
            const int ns = stage + 1 == stages ? 0 : stage + 1;
            const uint32_t nphase = ns == 0 ? phase ^ 1u : phase;
            const uint64_t soff = (uint64_t)((uint32_t)stage * (uint32_t)(STAGE_BYTES >> 4));  // stays inside the address field
            const uint32_t eb = empty0 + (uint32_t)stage * 8u, ebp = empty0_peer + (uint32_t)stage * 8u;
            const uint32_t nf = full0 + (uint32_t)ns * 8u;
            const uint32_t first = kb > kc ? 1u : 0u;  // the chunk's first MMA overwrites the accumulator
            if (TERMS == 1)
              ready = ptx::kblock_f16<PAIR, A_STEP, B_STEP>(d_main, a_desc0[0] + soff, b_desc0[0] + soff, IDESC, first, eb,
                                                            ebp, nf, nphase);
            else  // hi * [hi | lo] into d_main (width 2 BN), lo * hi into d_tail
              ready = ptx::kblock_x3<TERMS == 2, A_STEP, B_STEP>(d_main, d_tail, a_desc0[0] + soff,
                                                                 a_desc0[NSPLIT - 1] + soff, b_desc0[0] + soff,
                                                                 b_desc0[0] + soff, IDESC_WIDE, IDESC, first, eb, nf,
                                                                 nphase);
            stage = ns;
            phase = nphase;
          }
          if (ok) {  // this chunk's accumulators are complete
            if (PAIR) {
              ptx::mma_commit_pair(ptx::smem_addr(&acc_full[buf]));
              ptx::mma_commit_pair(at_peer(&acc_full[buf]));
            } else {
              ptx::mma_commit(&acc_full[buf]);
            }
          }
        }
      }
      if (!ok) s_fail = 1;
    }
  } else {
    // ---------------- epilogue: warps 2..9 ----------------
    constexpr int HALF = BN / 2;
    const int quarter = warp & 3;        // the TMEM lanes this warp may read: 32*quarter .. +31
    const int half = (warp - 2) >> 2;    // which half of the tile's columns it takes
    const int ch0 = half * HALF;
    float unscale1 = 1.f, unscale2 = 1.f;  // fp16 pairs: the operands were scaled by powers of two
    if (TERMS == 2) f16_unscale(p.rec_a->scale_exp, p.rec_b->scale_exp, unscale1, unscale2);
    int use = 0;
    uint32_t epi_phase = 0;
    bool ok = true;
    // the epilogue warps' own rendezvous: an mbarrier, so that this wait is bounded like every other
    auto epi_sync = [&]() -> bool {
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&epi_bar);
      const bool done = ptx::mbar_wait_relaxed(&epi_bar, epi_phase, 32);
      epi_phase ^= 1;
      return done;
    };
    TilePieces pieces(p.streamk, p.units, p.num_k, total_tiles, worker, p.workers, p.sk_first, p.sk_workers);
    int tile, kb0, kb1;
    while (ok && pieces.next(tile, kb0, kb1)) {
      const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);

      // Finishes and stores N columns of this thread's row, from column c of the warp's half on. A tile's
      // epilogue runs once, so its code is as good as never in the instruction caches when it starts: what
      // it costs is its length. Bias, activation and the kinds of store are therefore chosen outside the
      // loops, and nothing is repeated per element. (Chosen per element it was some 4,000 instructions, and
      // 19600 x 288 x 64, two k-blocks per tile, had ten warps waiting for code for each one that issued;
      // the convolution's backward pass that this product belongs to went from 150 to 120 us.)
      auto finish_store = [&](auto &v, auto size, int c) {
        constexpr int NV = decltype(size)::value;
        int bz, mb, nb;
        decode(tile, bz, mb, nb);
        const long long m = (long long)(PAIR ? mb * 2 + (int)rank : mb) * TC_BM + quarter * 32 + lane;
        const long long nbase = (long long)nb * BN + ch0 + c;
        if (m >= p.M || nbase >= (p.C_hi ? p.ld_split : p.N)) return;
        const int valid = p.N - nbase >= NV ? NV : (int)(p.N - nbase);  // may be <= 0 in front of a split's padding
        const float *bias = reinterpret_cast<const float *>(p.ep.bias);
        if (p.ep.bias_kind == B200_BIAS_COL) {
          if (valid == NV) {
#pragma unroll
            for (int j = 0; j < NV; ++j) v[j] = __fadd_rn(v[j], __ldg(bias + nbase + j));
          } else {
#pragma unroll
            for (int j = 0; j < NV; ++j)
              if (j < valid) v[j] = __fadd_rn(v[j], __ldg(bias + nbase + j));
          }
        } else if (p.ep.bias_kind == B200_BIAS_ROW) {
          const float bm = __ldg(bias + m);
#pragma unroll
          for (int j = 0; j < NV; ++j) v[j] = __fadd_rn(v[j], bm);
        }
        const float alpha = (float)p.ep.alpha;
        if (p.ep.act == B200_ACT_RECTIFY) {
#pragma unroll
          for (int j = 0; j < NV; ++j) v[j] = apply_act<float>(v[j], B200_ACT_RECTIFY, alpha);
        } else if (p.ep.act == B200_ACT_LEAKY) {
#pragma unroll
          for (int j = 0; j < NV; ++j) v[j] = apply_act<float>(v[j], B200_ACT_LEAKY, alpha);
        }
        if (p.C) {
          float *crow = reinterpret_cast<float *>(p.C) + (long long)bz * p.strideC + m * p.ldc + nbase;
          if (p.c_vec && valid == NV) {
            if (p.ep.accumulate) {  // Incr mode: the rounded result is added to what C holds
#pragma unroll
              for (int j = 0; j < NV; j += 4) {
                const float4 old = *reinterpret_cast<const float4 *>(crow + j);
                *reinterpret_cast<float4 *>(crow + j) = make_float4(__fadd_rn(old.x, v[j]), __fadd_rn(old.y, v[j + 1]),
                                                                    __fadd_rn(old.z, v[j + 2]), __fadd_rn(old.w, v[j + 3]));
              }
            } else {
#pragma unroll
              for (int j = 0; j < NV; j += 4)
                *reinterpret_cast<float4 *>(crow + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < NV; ++j)
              if (j < valid) crow[j] = p.ep.accumulate ? __fadd_rn(crow[j], v[j]) : v[j];
          }
        }
        if (p.C_hi) {
          // the result as the next product's A operand: TF32 head and tail, 16 bytes at a time;
          // columns between N and the pitch hold zeros
          float *hrow = p.C_hi + m * p.ld_split + nbase, *lrow = p.C_lo + m * p.ld_split + nbase;
#pragma unroll
          for (int j = 0; j < NV; j += 4) {
            if (nbase + j < p.ld_split) {
              float h[4], l[4];
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const float o = j + t < valid ? v[j + t] : 0.f;
                uint32_t hb;
                asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(o));
                h[t] = __uint_as_float(hb);
                asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hb) : "f"(__fsub_rn(o, h[t])));
                l[t] = __uint_as_float(hb);
              }
              *reinterpret_cast<float4 *>(hrow + j) = make_float4(h[0], h[1], h[2], h[3]);
              *reinterpret_cast<float4 *>(lrow + j) = make_float4(l[0], l[1], l[2], l[3]);
            }
          }
        }
      };

      if (TERMS == 1) {
        // one chunk per tile: straight from tensor memory to C
        const int buf = use & 1;
        const uint32_t acc_phase = (uint32_t)((use >> 1) & 1);
        ++use;
        if (!ptx::mbar_wait_relaxed(&acc_full[buf], acc_phase)) {
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
#pragma unroll 1
        for (int c = 0; c < HALF; c += 32) {
          uint32_t r[32];
          ptx::tmem_ld_32x32(lane_addr + (uint32_t)(buf * ACC_COLS + ch0 + c), r);
          ptx::tmem_ld_wait();
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          finish_store(v, std::integral_constant<int, 32>(), c);
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) ptx::mbar_arrive_cluster(at_leader(&acc_empty[buf]));
          else ptx::mbar_arrive(&acc_empty[buf]);
        }
      } else {
        // pairs: the tensor core adds into its accumulator with truncation, a bias that grows
        // with the length of the accumulation chain. Chains are therefore cut into k-chunks; each
        // chunk's two accumulators (main and cross terms) are folded here into fp32 registers
        // with round-to-nearest adds while the next chunk is being multiplied.
        float acc[TERMS != 1 ? HALF : 1];
#pragma unroll
        for (int j = 0; j < (TERMS != 1 ? HALF : 1); ++j) acc[j] = 0.f;
        for (int kc = kb0; kc < kb1 && ok; kc += p.chunk_k) {
          const int buf = use & 1;
          const uint32_t acc_phase = (uint32_t)((use >> 1) & 1);
          ++use;
          if (!ptx::mbar_wait_relaxed(&acc_full[buf], acc_phase)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
#pragma unroll
          for (int c = 0; c < (TERMS != 1 ? HALF : 0); c += 16) {
            uint32_t rm[16], rt[16];
            ptx::tmem_ld_32x16(lane_addr + (uint32_t)(buf * ACC_COLS + ch0 + c), rm);
            ptx::tmem_ld_32x16(lane_addr + (uint32_t)(buf * ACC_COLS + BN + ch0 + c), rt);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j)
              // the tails of fp16 pairs carry a factor of 2^11
              acc[c + j] = __fadd_rn(acc[c + j], __fadd_rn(__uint_as_float(rm[j]),
                                                           TERMS == 2 ? __fmul_rn(__uint_as_float(rt[j]), 4.8828125e-4f)
                                                                      : __uint_as_float(rt[j])));
          }
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&acc_empty[buf]);
        }
        if (kb0 != 0 || kb1 != p.num_k) {
          // part of a tile: leave it in the workspace; the CTA that delivers the last part finishes the tile
          constexpr int NACC = TERMS != 1 ? HALF : 1;
          const int tile_u0 = (tile - p.sk_first) * p.num_k;  // among the units that are shared out
          const size_t slot_floats = (size_t)TC_BM * BN;
          const size_t within = ((size_t)(warp - 2) * HALF) * 32 + lane;
          if (ok) {
            float *wsp = p.ws + (size_t)share_slot(worker, tile_u0, p.units, p.sk_workers) * slot_floats + within;
#pragma unroll
            for (int j = 0; j < NACC; ++j) __stcg(wsp + j * 32, acc[j]);
          } else {
            s_fail = 1;
          }
          __threadfence();
          const int c_first = share_of_unit(tile_u0, p.units, p.sk_workers);
          const int c_last = share_of_unit(tile_u0 + p.num_k - 1, p.units, p.sk_workers);
          bool met = epi_sync();
          if (warp == 2 && lane == 0) {
            s_last = (atomicAdd(p.tile_count + (tile - p.sk_first), 1) == c_last - c_first) ? 1 : 0;
            if (s_last) p.tile_count[tile - p.sk_first] = 0;  // zero again for the next launch
          }
          met = epi_sync() && met;
          if (!met || *(volatile int *)&s_fail) {
            ok = false;
            break;
          }
          if (!*(volatile int *)&s_last) continue;
          __threadfence();
#pragma unroll
          for (int j = 0; j < NACC; ++j) acc[j] = 0.f;
          // k order: CTA c's share precedes CTA c + 1's. On narrow tiles the loads of three parts are in
          // flight together (a part is a latency of about a microsecond); on wide ones there are no registers
          // for that, and one SM's share of the L2 rate is the bound.
          constexpr int PF = NACC == 32 ? 3 : 1;
          for (int c = c_first; c <= c_last; c += PF) {
            float part[PF][NACC];
#pragma unroll
            for (int q = 0; q < PF; ++q) {
              if (c + q <= c_last) {
                const float *src = p.ws + (size_t)share_slot(c + q, tile_u0, p.units, p.sk_workers) * slot_floats + within;
#pragma unroll
                for (int j = 0; j < NACC; ++j) part[q][j] = PF > 1 ? __ldcg(src + j * 32) : ptx::ld_cg_ordered(src + j * 32);
              } else {
#pragma unroll
                for (int j = 0; j < NACC; ++j) part[q][j] = 0.f;
              }
            }
#pragma unroll
            for (int q = 0; q < PF; ++q) {
              if (c + q <= c_last) {
#pragma unroll
                for (int j = 0; j < NACC; ++j) acc[j] = __fadd_rn(acc[j], part[q][j]);
              }
            }
          }
        }
        if (ok) {
          if (TERMS == 2) {
#pragma unroll
            for (int j = 0; j < (TERMS != 1 ? HALF : 1); ++j) acc[j] = __fmul_rn(__fmul_rn(acc[j], unscale1), unscale2);
          }
          finish_store(acc, std::integral_constant<int, TERMS != 1 ? HALF : 1>(), 0);
        }
      }
    }
    if (!ok) s_fail = 1;
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  // a pair: neither CTA leaves, or gives its tensor memory back, while the other may still read its
  // shared memory or arrive on its barriers (every wait above is bounded, so both get here)
  if (PAIR) ptx::cluster_sync();
  if (threadIdx.x == 0 && s_fail) atomicExch(p.err_flag, 1);
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    if (PAIR) ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else ptx::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------
// What the tensor cores can do with kind::tf32 when nothing else is in the way: every SM issues
// 128 x 256 x 8 MMAs back to back on operands that already sit in shared memory, with no loads
// and no epilogue. The rate it reaches is the denominator of the float32 tensor rooflines.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 1) tf32_peak_kernel(int batches, int *err_flag) {
  constexpr int BN = 256, PER_BATCH = 16;
  extern __shared__ __align__(1024) unsigned char pk_smem_raw[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tmem_base_s;
  unsigned char *smem = reinterpret_cast<unsigned char *>(((uintptr_t)pk_smem_raw + 1023) & ~(uintptr_t)1023);
  // operands: TF32 values of both signs and mixed magnitude (all-zero operands would flatter the clocks)
  uint32_t *w = reinterpret_cast<uint32_t *>(smem);
  for (int i = threadIdx.x; i < (TC_BM + BN) * TC_ROW_BYTES / 4; i += blockDim.x) {
    const uint32_t h = (uint32_t)i * 2654435761u + blockIdx.x * 40503u;
    w[i] = (h & 0x80000000u) | (0x3F000000u + ((h >> 3) & 0x00FFE000u));
  }
  ptx::fence_proxy_async_smem();
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    ptx::mbar_init(&bar[0], 1);
    ptx::mbar_init(&bar[1], 1);
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    ptx::tmem_alloc(&tmem_base_s, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  if (threadIdx.x == 0) {
    constexpr uint32_t IDESC = make_idesc(2, false, false, TC_BM, BN);
    const uint32_t sa = ptx::smem_addr(smem), sb = sa + TC_BM * TC_ROW_BYTES;
    bool ok = true;
    for (int b = 0; b < batches && ok; ++b) {
#pragma unroll
      for (int i = 0; i < PER_BATCH; ++i) {
        const uint32_t off = (uint32_t)(i & 3) * 32;  // the four 8-wide k-slices of the 32-wide slab
        ptx::mma_tf32(tmem_base + (uint32_t)((i >> 2) & 1) * BN, make_smem_desc(sa + off, 16, 1024, 2),
                      make_smem_desc(sb + off, 16, 1024, 2), IDESC, (b | i) ? 1u : 0u);
      }
      ptx::mma_commit(&bar[b & 1]);
      // one batch stays in flight: wait for the batch before this one
      if (b > 0) ok = ptx::mbar_wait(&bar[(b - 1) & 1], (uint32_t)(((b - 1) >> 1) & 1));
    }
    if (ok && batches > 0) ok = ptx::mbar_wait(&bar[(batches - 1) & 1], (uint32_t)(((batches - 1) >> 1) & 1));
    if (!ok) atomicExch(err_flag, 1);
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)sym;
  });
  return fn;
}

// A 3-D map (contiguous dim, rows, batch) over a row-major matrix with `ld` elements per row.
int encode_map(b200_engine *e, CUtensorMap *map, int es, const void *base, long long inner, long long rows,
                      long long batch, long long ld, long long batch_stride, int box_inner, int box_rows,
                      bool atom32) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return set_error(e, B200_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * es, (cuuint64_t)(batch > 1 ? batch_stride : rows * ld) * es};
  cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, es == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                  const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  atom32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(e, B200_ERR_CUDA,
                     "cuTensorMapEncodeTiled failed (%d): dims %lld x %lld x %lld, ld %lld, box %d x %d", (int)r,
                     inner, rows, batch, ld, box_inner, box_rows);
  return B200_OK;
}

static bool tc_eligible(int dtype, long long M, long long N, long long K, long long lda, long long ldb,
                        long long ldc, long long batch, long long strideA, long long strideB, const void *A,
                        const void *B, const void *C) {
  if (dtype != B200_F32 && dtype != B200_BF16) return false;
  if (M < 1 || N < 1 || K < 1) return false;
  // tiny problems: a 128-row tile would be mostly padding and the launch is latency-bound anyway
  if (M * N * K < 64LL * 64 * 64) return false;
  // bf16 operands are read in place, so a narrow B cannot meet TMA's pitch rule; float32 operands
  // are re-pitched by the split pass and any N works (the tile is padded with zero columns)
  if (N < 16 && dtype == B200_BF16) return false;
  if (N < 16 && M < 128) return false;
  if ((uintptr_t)C % 4 != 0) return false;
  if (dtype == B200_BF16) {
    if (((uintptr_t)A | (uintptr_t)B) % 16 != 0) return false;
    // TMA reads the caller's buffers directly: row pitch and batch pitch in bytes must be 16-byte multiples
    if ((lda * 2) % 16 || (ldb * 2) % 16) return false;
    if (batch > 1 && ((strideA * 2) % 16 || (strideB * 2) % 16)) return false;
  }
  // float32 goes through the split pass, which re-pitches rows itself: no constraint on lda / ldb
  (void)ldc;
  return true;
}

// Bytes of one ring stage in one CTA (the kernel's STAGE_BYTES).
static size_t tc_stage_bytes(int terms, int bn, bool pair) {
  const size_t a = (size_t)TC_BM * TC_ROW_BYTES, b = (size_t)bn * TC_ROW_BYTES;
  return pair ? a + b / 2 : (terms == 1 ? 1 : 2) * (a + b);
}

// grid = CTAs; pairs launch as clusters of two.
template <int TERMS, int BN, bool A_MN, bool B_MN, bool PAIR>
static int launch_tc(b200_engine *e, const CUtensorMap *tm, const GemmTcParams &p, int grid) {
  auto kern = gemm_tc_kernel<TERMS, BN, A_MN, B_MN, PAIR>;
  const size_t smem = (size_t)p.stages * tc_stage_bytes(TERMS, BN, PAIR) + 1024;
  static std::atomic<int> attr_dev_mask{0};  // devices on which the attribute is set; engines on other threads share it
  if (!(attr_dev_mask & (1 << (e->device & 31)))) {
    // opt in to the large dynamic carve-out: what the SM offers minus this kernel's static part
    cudaFuncAttributes fa;
    B200_CHECK_CUDA(e, cudaFuncGetAttributes(&fa, kern));
    const size_t optin = std::min<size_t>(e->smem_optin, 227 * 1024);
    B200_CHECK_CUDA(e, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)(optin - fa.sharedSizeBytes)));
    attr_dev_mask |= 1 << (e->device & 31);
  }
  if (PAIR) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = e->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_kernel does
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // Only clusters that are resident together may share the tiles out evenly: a GPU whose SMs do
    // not all pair up would otherwise run the left-over clusters as a second round.
    static std::atomic<int> max_clusters[32];
    int mc = max_clusters[e->device & 31];
    if (mc == 0) {
      B200_CHECK_CUDA(e, cudaOccupancyMaxActiveClusters(&mc, kern, &cfg));
      if (mc < 1) return set_error(e, B200_ERR_CUDA, "gemm_tc_kernel: no pair of CTAs fits this device");
      max_clusters[e->device & 31] = mc;
    }
    GemmTcParams pp = p;
    pp.workers = std::min(p.workers, mc);
    cfg.gridDim = dim3((unsigned)(2 * pp.workers));
    cfg.numAttrs = 2;
    B200_CHECK_CUDA(e, cudaLaunchKernelEx(&cfg, kern, tm[0], tm[1], tm[2], tm[3], pp));
  } else {
    launch_kernel(e, kern, grid, TC_THREADS, smem, tm[0], tm[1], tm[2], tm[3], p);
  }
  B200_CHECK_LAUNCH(e, "gemm_tc_kernel");
  e->flags_dirty = true;
  return B200_OK;
}

template <int TERMS, int BN, bool PAIR = false>
static int launch_tc_layout(b200_engine *e, bool a_mn, bool b_mn, const CUtensorMap *tm, const GemmTcParams &p,
                            int grid) {
  if (!a_mn && !b_mn) return launch_tc<TERMS, BN, false, false, PAIR>(e, tm, p, grid);
  if (!a_mn && b_mn) return launch_tc<TERMS, BN, false, true, PAIR>(e, tm, p, grid);
  if (a_mn && !b_mn) return launch_tc<TERMS, BN, true, false, PAIR>(e, tm, p, grid);
  return launch_tc<TERMS, BN, true, true, PAIR>(e, tm, p, grid);
}


// Which of a float32 product's two launches this is, and what decides on the device whether it runs.
struct F16Gate {
  const F16Rec *rec_a = nullptr, *rec_b = nullptr;
  unsigned limit_a = 0, limit_b = 0;
  const int *redo = nullptr;
  F16Rec *clear_a = nullptr, *clear_b = nullptr;
};

// terms = 1 (bf16), 2 or 3 (fp32 split into head/tail, fp16 or TF32). a_mn / b_mn: the operand is stored
// with its m / n index contiguous (see the file comment).
int gemm_tc_core(b200_engine *e, int terms, bool a_mn, bool b_mn, long long M, long long N, long long K,
                 const TcOperand &a, const TcOperand &b, void *C, long long ldc, long long batch, long long strideC,
                 const Epilogue &ep, float *C_hi = nullptr, float *C_lo = nullptr, long long ld_split = 0,
                 const F16Gate &gate = F16Gate()) {
  const int es = terms == 3 ? 4 : 2;
  const int bk = TC_ROW_BYTES / es;
  // tile width: the widest that still gives every SM a tile, to keep small problems spread out
  const int tiles_m = (int)((M + TC_BM - 1) / TC_BM);
  const bool may_share_k = terms != 1 && !(e->flags & B200_ENGINE_NO_STREAMK);
  int bn = terms == 1 ? 256 : 128;
  // tile width: the widest that still gives every SM a tile. A problem too small for that gets the
  // narrow tiles whether or not its k range is shared out as well: one SM pulls operands from L2 at a
  // fixed rate, so more CTAs on more SMs shorten the k loop of each
  while (bn > 64 && (long long)tiles_m * ((N + bn - 1) / bn) * batch < e->sm_count) bn /= 2;
  while (bn > 64 && bn / 2 >= N) bn /= 2;
  const int tiles_n = (int)((N + bn - 1) / bn);
  // CTA pairs on 256-row tiles (bf16), when the widest tiles are in use and there are enough of
  // them to keep every pair busy for several rounds (a pair's tile is twice the size: the last
  // round's idle time doubles with it)
  const int pairs = e->sm_count / 2;
  const long long pair_tiles = (M + 2 * TC_BM - 1) / (2 * TC_BM) * tiles_n * batch;
  const bool pair = !(e->flags & B200_ENGINE_NO_PAIRS) && terms == 1 && bn == 256 && pair_tiles >= 4LL * pairs;

  CUtensorMap tm[4];
  memset(tm, 0, sizeof tm);
  const int mn_box = TC_ROW_BYTES / es;
  const long long a_batch = a.shared ? 1 : batch, b_batch = b.shared ? 1 : batch;
  for (int h = 0; h < (terms == 1 ? 1 : 2); ++h) {
    const void *ap = h == 0 ? a.p0 : a.p1, *bp = h == 0 ? b.p0 : b.p1;
    int rc;
    if (!a_mn)
      rc = encode_map(e, &tm[h], es, ap, K, M, a_batch, a.ld, a.batch_stride, bk, TC_BM, false);
    else
      rc = encode_map(e, &tm[h], es, ap, M, K, a_batch, a.ld, a.batch_stride, mn_box, bk, es == 4);
    if (rc != B200_OK) return rc;
    if (!b_mn)  // a pair's bf16 CTAs load half of the tile's B rows each
      rc = encode_map(e, &tm[2 + h], es, bp, K, N, b_batch, b.ld, b.batch_stride, bk,
                      pair ? bn / 2 : bn, false);
    else
      rc = encode_map(e, &tm[2 + h], es, bp, N, K, b_batch, b.ld, b.batch_stride, mn_box, bk, es == 4);
    if (rc != B200_OK) return rc;
  }
  if (terms == 1) {
    tm[1] = tm[0];
    tm[3] = tm[2];
  }

  GemmTcParams p;
  p.M = M;
  p.N = N;
  p.K = K;
  p.batch = batch;
  p.C = C;
  p.ldc = ldc;
  p.strideC = strideC;
  p.C_hi = C_hi;
  p.C_lo = C_lo;
  p.ld_split = ld_split;
  p.tiles_m = tiles_m;
  p.tiles_n = tiles_n;
  p.num_k = (int)((K + bk - 1) / bk);
  // bf16: one chain per tile. TF32 pairs: 8 k-blocks = 256 k = 32 accumulation steps per chain, which keeps
  // the truncation bias of the tensor core's adder near 5e-7 relative (4096^3: 6.4e-7 of the result's norm in
  // all). fp16 pairs: 6 k-blocks = 384 k = 24 steps: 5.0e-7 at 401 us; 8 blocks 6.5e-7 at 396, 4 blocks
  // 3.6e-7 at 413.
  p.chunk_k = terms == 1 ? p.num_k : (terms == 2 ? 6 : 8);
  p.rec_a = gate.rec_a;
  p.rec_b = gate.rec_b;
  p.limit_a = gate.limit_a;
  p.limit_b = gate.limit_b;
  p.redo = gate.redo;
  p.clear_a = gate.clear_a;
  p.clear_b = gate.clear_b;
  p.group_m = std::min(tiles_m, 8);
  p.c_vec = (C && ldc % 4 == 0 && (uintptr_t)C % 16 == 0 && (batch == 1 || strideC % 4 == 0)) ? 1 : 0;
  p.a_zmul = a.shared ? 0 : 1;
  p.b_zmul = b.shared ? 0 : 1;
  p.ep = ep;
  p.err_flag = e->d_flags + 2;
  const size_t stage_bytes = tc_stage_bytes(terms, bn, pair);
  const size_t budget = std::min<size_t>(e->smem_optin, 227 * 1024) - 4096;  // static part + alignment slack
  p.stages = (int)std::max<size_t>(2, std::min<size_t>(8, budget / stage_bytes));
  const long long total_tiles = (long long)tiles_m * tiles_n * batch;
  if (total_tiles >= (1LL << 31))
    return set_error(e, B200_ERR_UNSUPPORTED, "b200_gemm: %lld output tiles are more than one launch takes", total_tiles);
  int grid = (int)std::min<long long>(total_tiles, e->sm_count);
  p.streamk = 0;
  p.units = 0;
  p.ws = nullptr;
  p.tile_count = nullptr;
  p.workers = grid;
  p.sk_first = 0;
  p.sk_workers = grid;
  if (pair) {
    p.tiles_m = (int)((M + 2 * TC_BM - 1) / (2 * TC_BM));
    p.group_m = std::min(p.tiles_m, 4);  // the same 8 x 128 rows of A per raster group
    p.workers = (int)std::min<long long>(pair_tiles, pairs);
    return launch_tc_layout<1, 256, true>(e, a_mn, b_mn, tm, p, 2 * p.workers);
  }

  if (terms == 1) {
    if (bn == 256) return launch_tc_layout<1, 256>(e, a_mn, b_mn, tm, p, grid);
    if (bn == 128) return launch_tc_layout<1, 128>(e, a_mn, b_mn, tm, p, grid);
    return launch_tc_layout<1, 64>(e, a_mn, b_mn, tm, p, grid);
  }
  // whole tiles per CTA would leave SMs idle: share out the k range instead (TilePieces)
  void *ws = nullptr;
  int sk_grid = grid;
  if (may_share_k && total_tiles <= b200_engine::kSkCounters &&
      streamk_pays(total_tiles, p.num_k, e->sm_count, &sk_grid)) {
    if (b200_get(e, 2LL * sk_grid * TC_BM * bn * 4, &ws) == B200_OK) {
      p.streamk = 1;
      p.units = (int)(total_tiles * p.num_k);  // small: k sharing is for launches of few tiles
      grid = sk_grid;
      p.workers = grid;
      p.sk_workers = grid;
      p.tile_count = e->sk_counters;
      p.ws = (float *)ws;
    }  // else: no room for the partial tiles, whole tiles per CTA
  } else if (int first = 0, sk = 0; may_share_k && total_tiles - total_tiles / e->sm_count * e->sm_count <= b200_engine::kSkCounters &&
                                    streamk_tail_pays(total_tiles, p.num_k, e->sm_count, &first, &sk)) {
    // several waves of tiles and a ragged last one: the full waves whole, the rest along k
    if (b200_get(e, 2LL * sk * TC_BM * bn * 4, &ws) == B200_OK) {
      p.streamk = 1;
      p.sk_first = first;
      p.sk_workers = sk;
      p.units = (int)((total_tiles - first) * p.num_k);
      p.tile_count = e->sk_counters;
      p.ws = (float *)ws;
    }
  }
  int rc;
  if (terms == 2)
    rc = bn == 128 ? launch_tc_layout<2, 128>(e, a_mn, b_mn, tm, p, grid)
                   : launch_tc_layout<2, 64>(e, a_mn, b_mn, tm, p, grid);
  else
    rc = bn == 128 ? launch_tc_layout<3, 128>(e, a_mn, b_mn, tm, p, grid)
                   : launch_tc_layout<3, 64>(e, a_mn, b_mn, tm, p, grid);
  if (ws) b200_put(e, ws, 0);  // stream order: whoever gets the block next runs after this kernel
  return rc;
}

// What a constant's split is kept under besides its extents: which slices of the buffer a batch reads.
static long long slice_stride(long long batch, long long stride) { return batch > 1 ? stride : 0; }

// Finds or makes room for the TF32 head and tail of a row-major fp32 matrix (rows x cols, pitch ld,
// `batch` of them), with a pitch that is a multiple of 4 elements. What is left to do is put into *job
// (job->src stays null if a constant's split was there already); blk_hi / blk_lo are the blocks that the
// caller hands back with b200_put once the consuming kernel has been launched.
static int plan_split_tf32(b200_engine *e, const float *src, long long rows, long long cols, long long ld,
                           long long batch, long long batch_stride, TcOperand *out, SplitJob *job, void **blk_hi,
                           void **blk_lo) {
  const long long ldo = (cols + 3) / 4 * 4;
  const long long elems = rows * ldo * batch;
  *blk_hi = *blk_lo = nullptr;
  out->ld = ldo;
  out->batch_stride = rows * ldo;
  out->shared = false;
  // a buffer declared constant (weights) is split once; the split is kept until the buffer is
  // released or un-declared, and the caller gets no blocks to hand back
  if (is_constant(e, src)) {
    if (CachedSplit *c = find_cached(e, src, 0, rows, cols, batch, ld, slice_stride(batch, batch_stride))) {
      out->p0 = c->hi;
      out->p1 = c->lo;
      out->ld = c->ld_out;
      return B200_OK;
    }
  }
  int rc = b200_get(e, elems * 4, blk_hi);
  if (rc != B200_OK) return rc;
  rc = b200_get(e, elems * 4, blk_lo);
  if (rc != B200_OK) {
    b200_put(e, *blk_hi, 0);
    *blk_hi = nullptr;
    return rc;
  }
  out->p0 = *blk_hi;
  out->p1 = *blk_lo;
  job->src = src;
  job->ld = ld;
  job->stride = batch_stride;
  job->rows = rows;
  job->cols = cols;
  job->batch = batch;
  job->hi = *blk_hi;
  job->lo = *blk_lo;
  job->ldo = ldo;
  return B200_OK;
}
// Once the split has been launched: a constant's is kept, and the blocks are no longer the caller's.
static void keep_split_tf32(b200_engine *e, const SplitJob &job, void **blk_hi, void **blk_lo) {
  if (!job.src || !is_constant(e, job.src)) return;
  add_cached(e, job.src, CachedSplit{0, job.rows, job.cols, job.batch, job.ld, *blk_hi, *blk_lo, job.ldo,
                                   slice_stride(job.batch, job.stride)});
  *blk_hi = *blk_lo = nullptr;
}

// The TF32 split of one operand (conv_tc.cu).
int split_operand_tf32(b200_engine *e, const float *src, long long rows, long long cols, long long ld,
                       long long batch, long long batch_stride, TcOperand *out, void **blk_hi, void **blk_lo) {
  SplitJob job;
  int rc = plan_split_tf32(e, src, rows, cols, ld, batch, batch_stride, out, &job, blk_hi, blk_lo);
  if (rc == B200_OK && job.src) rc = launch_split_tf32(e, job, SplitJob());
  if (rc == B200_OK) {
    keep_split_tf32(e, job, blk_hi, blk_lo);
    return B200_OK;
  }
  for (void **b : {blk_hi, blk_lo})
    if (*b) {
      b200_put(e, *b, 0);
      *b = nullptr;
    }
  return rc;
}

// One float32 operand of a product: A or B as it is stored.
struct F32Operand {
  const float *src;
  long long rows, cols, ld, batch, stride;
};

// The product from TF32 pairs. a_given: A is already split (TcOperand filled in).
static int gemm_f32_tf32(b200_engine *e, bool a_mn, bool b_mn, long long M, long long N, long long K,
                         const F32Operand *A, const TcOperand *a_given, const F32Operand &B, void *C, long long ldc,
                         long long batch, long long strideC, const Epilogue &ep, float *C_hi = nullptr,
                         float *C_lo = nullptr, long long ld_split = 0) {
  TcOperand a, b;
  SplitJob ja, jb;
  void *blk[4] = {nullptr, nullptr, nullptr, nullptr};
  int rc = B200_OK;
  if (a_given) a = *a_given;
  else rc = plan_split_tf32(e, A->src, A->rows, A->cols, A->ld, A->batch, A->stride, &a, &ja, &blk[0], &blk[1]);
  if (rc == B200_OK) rc = plan_split_tf32(e, B.src, B.rows, B.cols, B.ld, B.batch, B.stride, &b, &jb, &blk[2], &blk[3]);
  // one launch for both, but a constant's split, which is made once, is a launch of its own
  if (rc == B200_OK && B.src && is_constant(e, B.src)) {
    rc = launch_split_tf32(e, ja, SplitJob());
    if (rc == B200_OK) rc = launch_split_tf32(e, jb, SplitJob());
  } else if (rc == B200_OK) {
    rc = launch_split_tf32(e, ja, jb);
  }
  if (rc == B200_OK) {
    keep_split_tf32(e, ja, &blk[0], &blk[1]);
    // one matrix as both operands: only one of two equal entries is kept
    if (!(jb.src && is_constant(e, jb.src) && find_cached(e, jb.src, 0, jb.rows, jb.cols, jb.batch, jb.ld, slice_stride(jb.batch, jb.stride))))
      keep_split_tf32(e, jb, &blk[2], &blk[3]);
    rc = gemm_tc_core(e, 3, a_mn, b_mn, M, N, K, a, b, C, ldc, batch, strideC, ep, C_hi, C_lo, ld_split);
  }
  // stream order makes handing the scratch back safe: later users run after this kernel
  for (void *s2 : blk)
    if (s2) b200_put(e, s2, 0);
  return rc;
}

// One operand on its way to fp16 pairs (pitch a multiple of 8 values).
struct F16Operand {
  TcOperand op;
  SplitJob job;             // job.src stays null if a constant's pairs were there already
  F16Rec *rec = nullptr;
  void *blk[2] = {nullptr, nullptr};   // the TF32 pairs' place; a temporary operand's fp16 pairs lie in it too
  void *kept[2] = {nullptr, nullptr};  // a constant's record and heads, and its tails, before they are kept
};

// Finds a constant's pairs or takes room for an operand's. Nothing is launched and nothing kept here: what was
// taken is the caller's to hand back, also after an error.
// The blocks are as large as the TF32 pairs need, which take their place if the fp16 pairs turn out unusable.
// along_rows: the product sums along the rows as they are stored (else down the columns). A constant's pairs are
// kept for products of either kind.
static int plan_split_f16(b200_engine *e, const F32Operand &x, bool along_rows, F16Rec *scratch_rec, F16Operand *o) {
  const long long ldo = (x.cols + 7) / 8 * 8, elems = x.rows * ldo * x.batch;
  o->op.ld = ldo;
  o->op.batch_stride = x.rows * ldo;
  o->op.shared = false;
  int rc = B200_OK;
  const bool constant = is_constant(e, x.src);
  if (constant) {
    if (CachedSplit *c = find_cached(e, x.src, 2, x.rows, x.cols, x.batch, x.ld, slice_stride(x.batch, x.stride))) {
      o->rec = (F16Rec *)c->hi;
      o->op.p1 = c->lo;
    } else {
      rc = b200_get(e, 256 + elems * 2, &o->kept[0]);
      if (rc == B200_OK) rc = b200_get(e, elems * 2, &o->kept[1]);
      o->rec = (F16Rec *)o->kept[0];
      o->op.p1 = o->kept[1];
      o->job.src = x.src;
    }
    o->op.p0 = (char *)o->rec + 256;
  } else {
    o->rec = scratch_rec;
    o->job.src = x.src;
  }
  for (int h = 0; h < 2 && rc == B200_OK; ++h) rc = b200_get(e, elems * 4, &o->blk[h]);
  if (rc != B200_OK) return rc;
  if (!constant) {
    o->op.p0 = o->blk[0];
    o->op.p1 = o->blk[1];
  }
  o->job.ld = x.ld;
  o->job.stride = x.stride;
  o->job.rows = x.rows;
  o->job.cols = x.cols;
  o->job.batch = x.batch;
  o->job.hi = const_cast<void *>(o->op.p0);
  o->job.lo = const_cast<void *>(o->op.p1);
  o->job.ldo = ldo;
  o->job.rec = o->rec;
  o->job.limit = f16_small_limit(x.rows * x.cols * x.batch);
  o->job.lines = constant ? kLineRows | kLineCols : (along_rows ? kLineRows : kLineCols);
  return B200_OK;
}

// Once its split has been launched: a constant's pairs are kept, unless an equal entry (one matrix as both
// operands) is there already.
static void keep_split_f16(b200_engine *e, const F32Operand &x, F16Operand *o) {
  if (!o->kept[0] || find_cached(e, x.src, 2, x.rows, x.cols, x.batch, x.ld, slice_stride(x.batch, x.stride))) return;
  add_cached(e, x.src, CachedSplit{2, x.rows, x.cols, x.batch, x.ld, o->kept[0], o->kept[1], o->op.ld,
                                 slice_stride(x.batch, x.stride)});
  o->kept[0] = o->kept[1] = nullptr;
}

// Whether a product is worth fp16 pairs. They save about half of the 2 M N K / 200 TFLOP/s that TF32 pairs
// take; finding the largest magnitudes reads both operands once more (5 TB/s), and the launches that find
// nothing to do cost 8 us. Measured both ways (TF32 / fp16, us): 1024^3 26 / 27, 1000 x 1152 x 625 20 / 25, 1536^3
// 62 / 51, 2048 x 2048 x 1024 54 / 47, 8192 x 625 x 1152 112 / 100; with a constant B 25 / 24, 20 / 23, 58 / 45,
// 50 / 41, 111 / 99. The line lies between the second and the third. Not where a result may not depend on the batch: this rule, the scale and the way back
// all do.
static bool f16_pays(b200_engine *e, long long M, long long N, long long K, long long batch, const F32Operand &A,
                     const F32Operand &B) {
  if (e->flags & B200_ENGINE_NO_STREAMK) return false;
  const double saves = (double)M * N * K * batch / 200e12;
  const double reads = ((is_constant(e, A.src) ? 0.0 : (double)M * K) + (is_constant(e, B.src) ? 0.0 : (double)N * K)) * 4.0 * batch / 5e12;
  return saves > 1.3 * (reads + 8e-6);
}

// The product from fp16 pairs, with the TF32 launches behind it that run only if the pairs are unusable.
static int gemm_f32_f16(b200_engine *e, bool a_mn, bool b_mn, long long M, long long N, long long K,
                        const F32Operand &A, const F32Operand &B, void *C, long long ldc, long long batch,
                        long long strideC, const Epilogue &ep, float *C_hi = nullptr, float *C_lo = nullptr,
                        long long ld_split = 0) {
  F16Operand a, b;
  const F32Operand *xs[2] = {&A, &B};
  F16Operand *ops[2] = {&a, &b};
  int rc = plan_split_f16(e, A, !a_mn, e->f16_recs, &a);
  if (rc == B200_OK) rc = plan_split_f16(e, B, !b_mn, e->f16_recs + 1, &b);
  for (F16Operand *o : ops)
    if (rc == B200_OK && o->kept[0] && cudaMemsetAsync(o->rec, 0, sizeof(F16Rec), e->stream) != cudaSuccess)
      rc = set_error(e, B200_ERR_CUDA, "b200_gemm: clearing a record failed");
  const unsigned la = a.job.limit, lb = b.job.limit;
  if (rc == B200_OK && a.job.src) rc = launch_split_f16(e, a.job, b.job);
  else if (rc == B200_OK && b.job.src) rc = launch_split_f16(e, b.job, SplitJob());
  if (rc == B200_OK)
    for (int i = 0; i < 2; ++i) keep_split_f16(e, *xs[i], ops[i]);
  F16Gate gate;
  gate.rec_a = a.rec;
  gate.rec_b = b.rec;
  gate.limit_a = la;
  gate.limit_b = lb;
  if (rc == B200_OK)
    rc = gemm_tc_core(e, 2, a_mn, b_mn, M, N, K, a.op, b.op, C, ldc, batch, strideC, ep, C_hi, C_lo, ld_split, gate);
  if (rc == B200_OK) {
    TcOperand t[2];
    for (int i = 0; i < 2; ++i) {
      SplitJob &j = ops[i]->job;
      j.src = xs[i]->src;
      j.hi = ops[i]->blk[0];
      j.lo = ops[i]->blk[1];
      j.ldo = (xs[i]->cols + 3) / 4 * 4;
      t[i].p0 = j.hi;
      t[i].p1 = j.lo;
      t[i].ld = j.ldo;
      t[i].batch_stride = xs[i]->rows * j.ldo;
    }
    F16Gate redo;
    redo.redo = (int *)(e->f16_recs + 2);
    redo.clear_a = a.rec == e->f16_recs ? a.rec : nullptr;
    redo.clear_b = b.rec == e->f16_recs + 1 ? b.rec : nullptr;
    rc = launch_split_tf32_redo(e, a.job, b.job, a.rec, la, b.rec, lb, (int *)(e->f16_recs + 2));
    if (rc == B200_OK)
      rc = gemm_tc_core(e, 3, a_mn, b_mn, M, N, K, t[0], t[1], C, ldc, batch, strideC, ep, C_hi, C_lo, ld_split, redo);
  }
  if (rc != B200_OK) clear_f16_recs(e);
  // stream order makes handing the blocks back safe, also those whose kernels are queued
  for (F16Operand *o : ops)
    for (void *s2 : {o->blk[0], o->blk[1], o->kept[0], o->kept[1]})
      if (s2) b200_put(e, s2, 0);
  return rc;
}

static int gemm_tc(b200_engine *e, int dtype, int transA, int transB, long long M, long long N, long long K,
                   const void *A, long long lda, const void *B, long long ldb, void *C, long long ldc,
                   long long batch, long long strideA, long long strideB, long long strideC, const Epilogue &ep) {
  const bool a_mn = transA != 0;   // stored K x M: m contiguous
  const bool b_mn = transB == 0;   // stored K x N: n contiguous
  TcOperand a, b;
  if (dtype == B200_BF16) {
    a.p0 = A;
    a.ld = lda;
    a.batch_stride = strideA;
    b.p0 = B;
    b.ld = ldb;
    b.batch_stride = strideB;
    return gemm_tc_core(e, 1, a_mn, b_mn, M, N, K, a, b, C, ldc, batch, strideC, ep);
  }
  // stored shapes (rows x contiguous)
  const F32Operand fa{(const float *)A, transA ? K : M, transA ? M : K, lda, batch, strideA};
  const F32Operand fb{(const float *)B, transB ? N : K, transB ? K : N, ldb, batch, strideB};
  if (f16_pays(e, M, N, K, batch, fa, fb)) {
    const int rc = gemm_f32_f16(e, a_mn, b_mn, M, N, K, fa, fb, C, ldc, batch, strideC, ep);
    if (rc != B200_ERR_OOM) return rc;  // else: the TF32 pairs of constants may be there already
  }
  return gemm_f32_tf32(e, a_mn, b_mn, M, N, K, &fa, nullptr, fb, C, ldc, batch, strideC, ep);
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_gemm_chain(b200_engine *e, int transB, int64_t M, int64_t N, int64_t K, const void *A, const void *A_hi,
                    const void *A_lo, int64_t lda, const void *B, int64_t ldb, void *C, void *C_hi, void *C_lo,
                    int64_t ldc, int64_t ld_split, const b200_epilogue *epi) {
  if (!e) return B200_ERR_INVALID;
  std::lock_guard<std::recursive_mutex> lk(e->mu);
  B200_REQUIRE(e, M >= 0 && N > 0 && K > 0, "b200_gemm_chain: bad extent");
  B200_REQUIRE(e, (A_hi == nullptr) == (A_lo == nullptr) && (C_hi == nullptr) == (C_lo == nullptr),
               "b200_gemm_chain: a head needs its tail");
  B200_REQUIRE(e, A || A_hi, "b200_gemm_chain: no A");
  B200_REQUIRE(e, C || C_hi, "b200_gemm_chain: no output");
  B200_REQUIRE(e, B, "b200_gemm_chain: B is null");
  B200_REQUIRE(e, lda >= K && ldb >= (transB ? K : N) && (!C || ldc >= N), "b200_gemm_chain: leading dimension too small");
  B200_REQUIRE(e, !A_hi || (lda % 4 == 0 && ((uintptr_t)A_hi | (uintptr_t)A_lo) % 16 == 0),
               "b200_gemm_chain: a split A needs a pitch that is a multiple of 4 and 16-byte aligned pointers");
  B200_REQUIRE(e, !C_hi || (ld_split == (N + 3) / 4 * 4 && ((uintptr_t)C_hi | (uintptr_t)C_lo) % 16 == 0),
               "b200_gemm_chain: the split output needs the pitch N rounded up to a multiple of 4 and aligned pointers");
  if (epi) {
    B200_REQUIRE(e, epi->bias_kind >= 0 && epi->bias_kind <= 2 && epi->act >= 0 && epi->act <= 2,
                 "b200_gemm_chain: bad epilogue");
    B200_REQUIRE(e, epi->bias_kind == 0 || epi->bias != nullptr, "b200_gemm_chain: bias is null");
    B200_REQUIRE(e, epi->accumulate == 0, "b200_gemm_chain: accumulate cannot be combined with a chain");
  }
  if (M == 0) return B200_OK;
  DeviceGuard g(e);
  int rc = flush_pending(e);
  if (rc != B200_OK) return rc;
  const Epilogue ep = make_epilogue(epi);
  const void *probe = A ? A : A_hi;
  if (tc_eligible(B200_F32, M, N, K, lda, ldb, ldc, 1, 0, 0, probe, B, C ? C : C_hi)) {
    const F32Operand fa{(const float *)A, M, K, lda, 1, 0};
    const F32Operand fb{(const float *)B, transB ? N : K, transB ? K : N, ldb, 1, 0};
    TcOperand given;
    given.p0 = A_hi;
    given.p1 = A_lo;
    given.ld = lda;
    given.batch_stride = M * lda;
    if (!A_hi && f16_pays(e, M, N, K, 1, fa, fb)) {
      rc = gemm_f32_f16(e, false, transB == 0, M, N, K, fa, fb, C, ldc, 1, M * ldc, ep, (float *)C_hi, (float *)C_lo,
                        ld_split);
      if (rc != B200_ERR_OOM) return rc;
    }
    return gemm_f32_tf32(e, false, transB == 0, M, N, K, &fa, A_hi ? &given : nullptr, fb, C, ldc, 1, M * ldc, ep,
                         (float *)C_hi, (float *)C_lo, ld_split);
  }
  // small or oddly shaped: the plain product, then the rewrite pass; both need the tensors unsplit
  if (!A)
    return set_error(e, B200_ERR_UNSUPPORTED,
                     "b200_gemm_chain: this shape runs on the CUDA-core kernel, which reads an unsplit A; pass A");
  void *tmp = nullptr;
  float *cf = (float *)C;
  long long ldc_eff = ldc;
  if (!C) {
    rc = b200_get(e, M * N * 4, &tmp);
    if (rc != B200_OK) return rc;
    cf = (float *)tmp;
    ldc_eff = N;
  }
  rc = gemm_simt(e, B200_F32, 0, transB, M, N, K, A, lda, B, ldb, cf, ldc_eff, 1, 0, 0, 0, ep);
  if (rc == B200_OK && C_hi) {
    SplitJob job;
    job.src = cf;
    job.ld = ldc_eff;
    job.rows = M;
    job.cols = N;
    job.batch = 1;
    job.hi = C_hi;
    job.lo = C_lo;
    job.ldo = ld_split;
    rc = launch_split_tf32(e, job, SplitJob());
  }
  if (tmp) b200_put(e, tmp, 0);
  return rc;
}

int b200_tf32_peak(b200_engine *e, int batches, double *tflops) {
  if (!e) return B200_ERR_INVALID;
  std::lock_guard<std::recursive_mutex> lk(e->mu);
  B200_REQUIRE(e, tflops != nullptr, "b200_tf32_peak: null pointer");
  B200_REQUIRE(e, batches >= 1 && batches <= 1000000, "b200_tf32_peak: 1 .. 1000000 batches of 16 instructions");
  B200_NOT_WHILE_CAPTURING(e, "b200_tf32_peak");
  DeviceGuard g(e);
  int rc = flush_pending(e);
  if (rc != B200_OK) return rc;
  const size_t smem = (size_t)(TC_BM + 256) * TC_ROW_BYTES + 1024;
  B200_CHECK_CUDA(e, cudaFuncSetAttribute(tf32_peak_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaEvent_t ev0, ev1;
  B200_CHECK_CUDA(e, cudaEventCreate(&ev0));
  B200_CHECK_CUDA(e, cudaEventCreate(&ev1));
  float best = 0.f;
  for (int rep = 0; rep < 4 && rc == B200_OK; ++rep) {  // the first repetition warms up
    cudaEventRecord(ev0, e->stream);
    tf32_peak_kernel<<<e->sm_count, 128, smem, e->stream>>>(batches, e->d_flags + 2);
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) {
      rc = set_error(e, B200_ERR_CUDA, "launch of tf32_peak_kernel failed: %s", cudaGetErrorString(le));
      break;
    }
    e->launches++;
    e->flags_dirty = true;
    cudaEventRecord(ev1, e->stream);
    rc = sync_stream_checked(e);
    float ms = 0.f;
    if (rc == B200_OK && cudaEventElapsedTime(&ms, ev0, ev1) == cudaSuccess && rep > 0 && (best == 0.f || ms < best))
      best = ms;
  }
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  if (rc != B200_OK) return rc;
  const double flops = 2.0 * TC_BM * 256 * 8 * 16.0 * batches * e->sm_count;
  *tflops = best > 0.f ? flops / (best * 1e-3) / 1e12 : 0.0;
  return B200_OK;
}

int b200_gemm_path(b200_engine *e, int dtype, int transA, int transB, int64_t M, int64_t N, int64_t K, int64_t lda,
                   int64_t ldb, int64_t ldc, const void *A, const void *B, const void *C) {
  (void)e;
  (void)transA;
  (void)transB;
  return tc_eligible(dtype, M, N, K, lda, ldb, ldc, 1, 0, 0, A, B, C) ? 1 : 0;
}

int b200_gemm(b200_engine *e, int dtype, int transA, int transB, int64_t M, int64_t N, int64_t K, const void *A,
              int64_t lda, const void *B, int64_t ldb, void *C, int64_t ldc, int64_t batch, int64_t strideA,
              int64_t strideB, int64_t strideC, const b200_epilogue *epi) {
  if (!e) return B200_ERR_INVALID;
  std::lock_guard<std::recursive_mutex> lk(e->mu);
  B200_REQUIRE(e, dtype == B200_F32 || dtype == B200_F64 || dtype == B200_BF16, "b200_gemm: dtype %d not supported",
               dtype);
  B200_REQUIRE(e, M >= 0 && N >= 0 && K >= 0 && batch >= 0, "b200_gemm: negative extent");
  if (M == 0 || N == 0 || batch == 0) return B200_OK;
  B200_REQUIRE(e, C != nullptr, "b200_gemm: C is null");
  const int64_t a_cols = transA ? M : K, b_cols = transB ? K : N;
  B200_REQUIRE(e, lda >= a_cols && ldb >= b_cols && ldc >= N, "b200_gemm: leading dimension too small (%lld %lld %lld)",
               (long long)lda, (long long)ldb, (long long)ldc);
  if (epi) {
    B200_REQUIRE(e, epi->bias_kind >= 0 && epi->bias_kind <= 2 && epi->act >= 0 && epi->act <= 2,
                 "b200_gemm: bad epilogue");
    B200_REQUIRE(e, epi->bias_kind == 0 || epi->bias != nullptr, "b200_gemm: bias is null");
  }
  DeviceGuard g(e);
  int rc = flush_pending(e);
  if (rc != B200_OK) return rc;
  Epilogue ep = make_epilogue(epi);
  if (K == 0) {
    // empty sum: C = epilogue(0); the CUDA-core kernel handles it with a zero-trip k loop
    if (dtype == B200_BF16) return set_error(e, B200_ERR_UNSUPPORTED, "b200_gemm: bf16 with K = 0");
    return gemm_simt(e, dtype, transA, transB, M, N, 0, C, lda, C, ldb, C, ldc, batch, 0, 0, strideC, ep);
  }
  B200_REQUIRE(e, A && B, "b200_gemm: null operand");
  if (tc_eligible(dtype, M, N, K, lda, ldb, ldc, batch, strideA, strideB, A, B, C)) {
    rc = gemm_tc(e, dtype, transA, transB, M, N, K, A, lda, B, ldb, C, ldc, batch, strideA, strideB, strideC, ep);
    // The float32 tensor-core path keeps TF32 splits of both operands in arena scratch (about
    // 2 x (|A| + |B|) bytes). The reference's MatMul needs no workspace, so an arena too full for
    // the splits still gets its product, from the CUDA-core kernel, which needs none.
    if (rc != B200_ERR_OOM || dtype != B200_F32) return rc;
  }
  if (dtype == B200_BF16)
    return set_error(e, B200_ERR_UNSUPPORTED,
                     "b200_gemm: bf16 operands need 16-byte aligned bases and row pitches (lda %lld, ldb %lld) and "
                     "at least 64^3 work",
                     (long long)lda, (long long)ldb);
  return gemm_simt(e, dtype, transA, transB, M, N, K, A, lda, B, ldb, C, ldc, batch, strideA, strideB, strideC, ep);
}

}  // extern "C"
