// fp32 GEMM on the tcgen05 tensor cores: every fp32 operand is held as three
// bf16 planes that add up to it exactly (x = h + m + l, 8 + 8 + 8 mantissa
// bits, each plane rounded to nearest), and
//
//   a w  =  ah wh + (ah wm + am wh) + (am wm + ah wl + al wh)
//
// is formed by six bf16 MMAs with fp32 accumulation.  The three products left
// out (am wl, al wm, al wl) are together at most 2^-24 of |a w|, the rounding of
// one fp32 product.
//
//   acc[m, n] = sum_k A[m, k] * W[n, k]     A: 3 planes of (M, K), W: 3 planes of (N, K)
//
// The tensor core's accumulation does not round to nearest, so a sum over all of
// K in TMEM would drift (one-sided) by more than a chain of FFMAs does.  Each
// 64-wide K block therefore gets a TMEM accumulator of its own, in which the
// small products are added first and the four ah wh steps last; the epilogue
// warps fetch it and add it to fp32 registers (round to nearest, K / 64
// additions instead of K).  Measured against 64-bit sums the result is closer
// than the FFMA kernel's.
//
// Two CTAs (a cluster on neighbouring SMs) share a 256 x PBN tile with
// tcgen05.mma.cta_group::2 and walk tiles persistently: each CTA's warp 0 streams the
// planes of its 128 rows of A and its half of W with TMA (3-D boxes of 64 K x rows
// x 3 planes), two warps of the even CTA issue the 24 MMAs of every K block (blocks in turn, an elected lane
// of each, see mbar_wait_all), the epilogue warps of both add
// up the blocks and run the fused epilogue.  Four accumulators rotate, so the adds run
// under the MMAs of the following blocks.
//
// A block has its own accumulator, so no order is needed between the MMAs of the two warps; but each
// warp waits for its own blocks only, and the ring has three stages: the barriers that announce
// landed operands are laid out by operand_ring.h so that a warp sees every phase of those it waits on.
//
// K split: where one wave of tiles leaves half of the SMs without work, two CTA pairs
// (a cluster of four) share a tile, each takes half of K, and the second pair hands
// its sums to the first through distributed shared memory (the operand ring, idle
// by then) before the epilogue: a fixed order, no scratch memory, no second kernel.
// One dual block of 256 + 77 tokens 381 -> 337 us.
//
// What bounds it: the tensor pipe (six MMAs per K step) and the operand loads: a K
// block of a 256 x 128 tile is 1536 cycles of MMA for 72 KiB per CTA and takes 1740 to 1800.  Not
// kept: one-CTA tiles of 128 x 256 with 32-wide K blocks (64-byte rows, half of W's bytes more per
// MMA: tensor pipe 38 % busy); 256 x 256 tiles (3072 cycles of MMA took 4060: two stages of
// operands, two accumulators, and an epilogue of 128 columns per thread between tiles).
//
// Measured: 24-block model at 512 x 512 (1024 + 333 tokens) 14.7 ms, one dual block of 256 + 77 tokens 291 us (15.1 and
// 294 while lane 0 alone ran the loads and the MMAs, here and in attention_split.cu);
// with FFMA GEMMs and the SIMT attention 754 ms and 4.74 ms.  What single steps gave, in the order they were made
// (each against the commit before it; the attention changed in between): one-CTA tiles -> pairs 19.26 -> 17.57 ms
// and 454 -> 411 us; K split 381 -> 337 us; no cluster-scope release in the accumulator's hand-back
// 16.8 -> 15.7 ms; GELU 15.5 -> 15.2 ms; 128-wide tiles instead of 256 15.3 -> 15.1 ms.
#include <cuda.h>
#include <mutex>

#include "gemm_epilogue.cuh"
#include "kernels.h"
#include "operand_ring.h"
#include "ptx.cuh"
#include "split3.cuh"

namespace sd3 {

int encode_tmap_3d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t d0, uint64_t d1, uint64_t d2,
                   uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t box0, uint32_t box1, uint32_t box2);
int device_sm_count();

namespace {

using gemm_detail::GemmArgs;
using gemm_detail::map_row;
using gemm_detail::RowMap;
using gemm_detail::st_global_32B;

constexpr int S_BM = 128;              // rows of A per CTA (256 per pair)
constexpr int S_KB = 64;               // K elements per block (128-byte rows)
constexpr int S_A_PLANE = S_BM * 128;  // 16 KiB

template <int PBN>
struct SplitCfg {
  static constexpr int W_ROWS = PBN / 2;  // rows of W per CTA
  static constexpr int W_PLANE = W_ROWS * 128;
  static constexpr int STAGE_BYTES = 3 * (S_A_PLANE + W_PLANE);  // 72 / 60 KiB
  static constexpr int STAGES = 3;                               // 216 / 180 KiB
  static constexpr int NBUF = 4;                                 // TMEM accumulators
  static_assert(NBUF % 2 == 0, "an accumulator belongs to one of the two MMA-issuing warps");
  static constexpr int TMEM_COLS = NBUF * PBN;
  static constexpr int EPI_WARPS = PBN == 64 ? 4 : 8;
  static constexpr int CPW = 64;                     // accumulator columns per epilogue thread (split_epilogue_64)
  static constexpr int MMA2_WARP = 2 + EPI_WARPS;    // second MMA-issuing warp
  static constexpr int THREADS = 32 * (3 + EPI_WARPS);
  using Ring = OperandRing<STAGES, 2>;  // two MMA-issuing warps, an elected lane of each
  static constexpr int BAR_BYTES = (Ring::FULL_BARS + STAGES + 2 * NBUF) * 8 + 8;  // barriers, TMEM address, abort flag
  static_assert(BAR_BYTES <= 256, "barrier block");
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 256 + 1024;
};

// 0.5 x (1 + tanh(u)) = x / (1 + e^(-2u)),  u = sqrt(2/pi) (x + 0.044715 x^3): no cancellation for
// negative u, two MUFU operations where tanhf takes some thirty instructions (an epilogue thread
// has 64 of them between two tiles)
__device__ __forceinline__ float gelu_tanh_f32(float x) {
  const float t = x * fmaf(x * x, -2.0f * 1.4426950408889634f * 0.7978845608028654f * 0.044715f,
                           -2.0f * 1.4426950408889634f * 0.7978845608028654f);  // -2 u log2(e)
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return x * r;
}

// eight consecutive fp32 outputs / eight outputs as three planes (16-byte stores)
__device__ __forceinline__ void store8_f32(float* p, const float* v) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

// Fused epilogue of 64 consecutive accumulator columns of output row m; the row exists.
template <int EPI, int OUT>  // OUT: 0 bf16 (unpatchify only), 1 fp32, 2 three bf16 planes
__device__ __forceinline__ void split_epilogue_64(float* v, const RowMap& rm, int n_base, const GemmArgs& g) {
  const GemmEpilogue& e = g.epi;
  const int N = g.N;
  if (n_base >= N) return;
  if (e.bias) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (n_base + 4 * i < N) {
        const float4 t = *(reinterpret_cast<const float4*>(e.bias + n_base) + i);
        v[4 * i] += t.x; v[4 * i + 1] += t.y; v[4 * i + 2] += t.z; v[4 * i + 3] += t.w;
      }
    }
  }
  if constexpr (EPI == EPI_QKV_NORM) {
    if (e.do_norm && n_base < e.qk_cols) {  // head_dim 64: these columns are one head
      const float* w = (n_base < (e.qk_cols >> 1)) ? e.wq : e.wk;
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
      for (int j = 0; j < 64; j += 4) {
        s0 = fmaf(v[j], v[j], s0);
        s1 = fmaf(v[j + 1], v[j + 1], s1);
        s2 = fmaf(v[j + 2], v[j + 2], s2);
        s3 = fmaf(v[j + 3], v[j + 3], s3);
      }
      const float r = rsqrtf(((s0 + s1) + (s2 + s3)) * (1.0f / 64.0f) + e.eps);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float4 t = w ? *(reinterpret_cast<const float4*>(w) + i) : make_float4(1.f, 1.f, 1.f, 1.f);
        v[4 * i] = v[4 * i] * r * t.x;
        v[4 * i + 1] = v[4 * i + 1] * r * t.y;
        v[4 * i + 2] = v[4 * i + 2] * r * t.z;
        v[4 * i + 3] = v[4 * i + 3] * r * t.w;
      }
    }
  }
  if constexpr (EPI == EPI_BIAS_GELU) {
#pragma unroll
    for (int j = 0; j < 64; ++j) v[j] = gelu_tanh_f32(v[j]);
  }
  if constexpr (EPI == EPI_ADD_TABLE) {
    const float4* t4 = reinterpret_cast<const float4*>(e.table + static_cast<long>(rm.t_in) * N + n_base);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (n_base + 4 * i < N) {
        const float4 t = t4[i];
        v[4 * i] += t.x; v[4 * i + 1] += t.y; v[4 * i + 2] += t.z; v[4 * i + 3] += t.w;
      }
    }
  }
  if constexpr (EPI == EPI_UNPATCHIFY) {
    // m = (b, r, s) over the patch grid; n = ph * (p * C) + pw * C + c
    const int p = e.up_patch, C = e.up_cin;
    const int s = rm.t_in % e.up_w, r = rm.t_in / e.up_w;
    const long Wpix = static_cast<long>(e.up_w) * p, Hpix = static_cast<long>(e.up_h) * p;
#pragma unroll
    for (int j = 0; j < 64; ++j) {
      const int n = n_base + j;
      if (n < N) {
        const int c = n % C, pw = (n / C) % p, ph = n / (C * p);
        const long idx = ((static_cast<long>(rm.b) * C + c) * Hpix + (r * p + ph)) * Wpix + (s * p + pw);
        if constexpr (OUT == 1)
          static_cast<float*>(e.out)[idx] = v[j];
        else
          static_cast<bf16*>(e.out)[idx] = __float2bfloat16(v[j]);
      }
    }
    return;
  }
  const long base = rm.orow * e.ldo + n_base;
  if constexpr (EPI == EPI_GATE_RESID) {
    const float4* g4 = reinterpret_cast<const float4*>(e.gate + static_cast<long>(rm.b) * e.gate_stride + n_base);
    const float4* r4 = reinterpret_cast<const float4*>(e.resid + base);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (n_base + 4 * i < N) {
        const float4 t = g4[i], x = r4[i];
        v[4 * i] = x.x + t.x * v[4 * i];
        v[4 * i + 1] = x.y + t.y * v[4 * i + 1];
        v[4 * i + 2] = x.z + t.z * v[4 * i + 2];
        v[4 * i + 3] = x.w + t.w * v[4 * i + 3];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = n_base + 16 * i;
    float* o = v + 16 * i;
    if constexpr (OUT == 1) {
      float* p = static_cast<float*>(e.out) + base + 16 * i;
      if (g.wide_store && n + 16 <= N) {
#pragma unroll
        for (int h = 0; h < 16; h += 8)
          st_global_32B(p + h, __float_as_uint(o[h]), __float_as_uint(o[h + 1]), __float_as_uint(o[h + 2]),
                        __float_as_uint(o[h + 3]), __float_as_uint(o[h + 4]), __float_as_uint(o[h + 5]),
                        __float_as_uint(o[h + 6]), __float_as_uint(o[h + 7]));
      } else {
        if (n < N) store8_f32(p, o);
        if (n + 8 < N) store8_f32(p + 8, o + 8);
      }
    } else {
      uint32_t u[3][8];
#pragma unroll
      for (int j = 0; j < 8; ++j) split3_x2(o[2 * j], o[2 * j + 1], u[0][j], u[1][j], u[2][j]);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        bf16* p = static_cast<bf16*>(e.out) + q * e.out_plane + base + 16 * i;
        if (g.wide_store && n + 16 <= N) {
          st_global_32B(p, u[q][0], u[q][1], u[q][2], u[q][3], u[q][4], u[q][5], u[q][6], u[q][7]);
        } else {
          if (n < N) reinterpret_cast<uint4*>(p)[0] = make_uint4(u[q][0], u[q][1], u[q][2], u[q][3]);
          if (n + 8 < N) reinterpret_cast<uint4*>(p)[1] = make_uint4(u[q][4], u[q][5], u[q][6], u[q][7]);
        }
      }
    }
  }
}

// One problem of a (possibly grouped) launch
struct SplitProblem {
  CUtensorMap tmA, tmW;
  GemmArgs g;
};

template <int PBN, int EPI, int OUT, int KSPLIT>
__global__ void __cluster_dims__(2 * KSPLIT, 1, 1) __launch_bounds__(SplitCfg<PBN>::THREADS, 1)
gemm_split_tcgen05_kernel(const __grid_constant__ SplitProblem p0, const __grid_constant__ SplitProblem p1,
                          const __grid_constant__ SplitProblem p2, const int end0, const int end1,
                          const int num_tiles) {
  using Cfg = SplitCfg<PBN>;
  using Ring = typename Cfg::Ring;
  constexpr int STAGES = Cfg::STAGES, NBUF = Cfg::NBUF, CPW = Cfg::CPW;
  constexpr uint32_t IDESC = make_idesc(1, 1, 2 * S_BM, PBN, 0, 0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Ring::FULL_BARS;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + NBUF;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + NBUF);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // known uniform
  const int lane = threadIdx.x & 31;
  const uint32_t part = cluster_ctarank() >> 1;  // share of K (KSPLIT == 2)
  const uint32_t rank = cluster_ctarank() & 1;   // CTA of the pair, 0 = leader
  const uint32_t leader = cluster_ctarank() & ~1u;
  const uint16_t pair_mask = static_cast<uint16_t>(3u << leader);
  const int pair = blockIdx.x / (2 * KSPLIT);  // index of the pair (cluster) among those that walk the tiles
  const int num_pairs = gridDim.x / (2 * KSPLIT);

  if (threadIdx.x == 0) {
    for (int s = 0; s < Ring::FULL_BARS; ++s) mbar_init(&full_bar[s], 1);  // leader's expect_tx arrival; bytes of both CTAs
    for (int s = 0; s < STAGES; ++s) mbar_init(&empty_bar[s], 1);          // one multicast commit per use
    for (int a = 0; a < NBUF; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * Cfg::EPI_WARPS);  // epilogue warps of both CTAs (leader's copy is used)
    }
    *s_abort = 0;
    fence_barrier_init();
    prefetch_tmap(&p0.tmA);
    prefetch_tmap(&p0.tmW);
    if (end1 > end0) {
      prefetch_tmap(&p1.tmA);
      prefetch_tmap(&p1.tmW);
    }
    if (num_tiles > end1) {
      prefetch_tmap(&p2.tmA);
      prefetch_tmap(&p2.tmW);
    }
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are initialised before any remote signal
  tc_fence_after_sync();
  if (warp != 0) {  // the TMA producer waits after its first weight tiles
    grid_dep_wait();
    grid_dep_launch();
  }
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const WaitCtx wc{s_abort, p0.g.status};
  // tiles of 256 x PBN: the first problem's up to end0, the second's up to end1, the third's
  // K blocks of this pair (the same K for all problems)
  const int kb0 = KSPLIT == 2 && part == 1 ? (p0.g.k_blocks + 1) / 2 : 0;
  const int KB = (KSPLIT == 2 && part == 0 ? (p0.g.k_blocks + 1) / 2 : p0.g.k_blocks) - kb0;
  float acc[CPW];  // running sums of an epilogue thread

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------
    Ring ring;
    bool ok = true;
    const bool issuer = elect_one();
    const uint32_t smem_at = smem_u32(smem), full_local = smem_u32(full_bar), full_leader = map_to_cta(full_local, leader);
    // the weights of a stage; all its bytes (both CTAs) are credited to the leader's barrier
    auto load_w = [&](const CUtensorMap* tmW, const Ring& at, int kb, int n0) {
      if (rank == 0) mbar_expect_tx_at(full_local + 8 * at.full, 2 * Cfg::STAGE_BYTES);
      tma_load_3d_pair_at(smem_at + at.stage * Cfg::STAGE_BYTES + 3 * S_A_PLANE, tmW, full_leader + 8 * at.full,
                          (kb0 + kb) * S_KB, n0, 0);
    };
    int pre = 0;  // stages of the first tile whose weights are under way before the wait
    if (p0.g.epi.w_static) {
      const SplitProblem& pp = pair < end0 ? p0 : pair < end1 ? p1 : p2;
      const int lt = pair - (pair < end0 ? 0 : pair < end1 ? end0 : end1);
      Ring at;
      for (; pre < STAGES && pre < KB; ++pre, at.next())
        if (issuer) load_w(&pp.tmW, at, pre, (lt % pp.g.tiles_n) * PBN + static_cast<int>(rank) * Cfg::W_ROWS);
    }
    grid_dep_wait();
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      const SplitProblem& pp = tile < end0 ? p0 : tile < end1 ? p1 : p2;
      const int lt = tile - (tile < end0 ? 0 : tile < end1 ? end0 : end1);
      const int m0 = (lt / pp.g.tiles_n) * (2 * S_BM) + static_cast<int>(rank) * S_BM;
      const int n0 = (lt % pp.g.tiles_n) * PBN + static_cast<int>(rank) * Cfg::W_ROWS;
      for (int kb = 0; kb < KB; ++kb) {
        if (pre > 0) {
          --pre;
        } else {
          if (!mbar_wait_all(&empty_bar[ring.stage], ring.stage_parity ^ 1, wc, DEV_TIMEOUT_EMPTY)) { ok = false; break; }
          if (issuer) load_w(&pp.tmW, ring, kb, n0);
        }
        if (issuer)
          tma_load_3d_pair_at(smem_at + ring.stage * Cfg::STAGE_BYTES, &pp.tmA, full_leader + 8 * ring.full,
                              (kb0 + kb) * S_KB, m0, 0);
        ring.next();
      }
    }
  } else if (warp == 1 || warp == Cfg::MMA2_WARP) {
    // ------------------------------ MMA issuers (leader only, two warps) ------
    if (rank == 0) {
      const int me = warp == 1 ? 0 : 1;
      Ring ring;
      int buf = 0;  // four accumulators: a warp sees every use of its two
      uint32_t bphase = 0;
      bool ok = true;
      const bool issuer = elect_one();
      const uint64_t desc0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        for (int kb = 0; kb < KB; ++kb) {
          if (ring.turn == me) {
            if (!mbar_wait_all(&tempty_bar[buf], bphase ^ 1, wc, DEV_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
            if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[ring.full], ring.full_parity, wc, DEV_TIMEOUT_FULL))) { ok = false; break; }
            tc_fence_after_sync();
            if (issuer) {
              const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * PBN);
              const uint64_t a0 = desc0 + static_cast<uint32_t>(ring.stage * (Cfg::STAGE_BYTES >> 4));
              const uint64_t w0 = a0 + (3 * S_A_PLANE >> 4);
              constexpr uint64_t AP = S_A_PLANE >> 4, WP = Cfg::W_PLANE >> 4;
              // (A plane, W plane), smallest products first
              constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
              for (int q = 0; q < 6; ++q)
#pragma unroll
                for (int k = 0; k < S_KB / 16; ++k)
                  mma_f16_ss_pair(d_tmem, a0 + PA[q] * AP + 2 * k, w0 + PW[q] * WP + 2 * k, IDESC, (q | k) != 0);
              mma_commit_pair(&empty_bar[ring.stage], pair_mask);  // frees the stage in both CTAs
              mma_commit_pair(&tfull_bar[buf], pair_mask);         // block sum ready in both CTAs
            }
          }
          ring.next();
          if (++buf == NBUF) { buf = 0; bphase ^= 1; }
        }
      }
    }
  } else if (warp >= 2 && warp < 2 + Cfg::EPI_WARPS) {
    // ------------------------------ accumulation + epilogue (both CTAs) -------
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = static_cast<int>(rank) * S_BM + quad * 32 + lane;
    int buf = 0;
    uint32_t bphase = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      const GemmArgs& g = tile < end0 ? p0.g : tile < end1 ? p1.g : p2.g;
      const int lt = tile - (tile < end0 ? 0 : tile < end1 ? end0 : end1);
      const int m = (lt / g.tiles_n) * (2 * S_BM) + row;
      const int n0 = (lt % g.tiles_n) * PBN + half * CPW;
#pragma unroll
      for (int j = 0; j < CPW; ++j) acc[j] = 0.f;
      for (int kb = 0; kb < KB; ++kb) {
        if (!mbar_wait_warp(&tfull_bar[buf], bphase, wc, DEV_TIMEOUT_TMEM_FULL)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) +
                               static_cast<uint32_t>(buf * PBN + half * CPW);
#pragma unroll
        for (int s = 0; s < CPW / 32; ++s) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_row + s * 32, r);
          tmem_wait_ld();
          if (s == CPW / 32 - 1) {  // everything is in registers: the accumulator may be reused
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[buf]), leader));
          }
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 t = __fadd2_rn(make_float2(acc[s * 32 + j], acc[s * 32 + j + 1]),
                                        make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])));
            acc[s * 32 + j] = t.x;
            acc[s * 32 + j + 1] = t.y;
          }
        }
        if (++buf == NBUF) { buf = 0; bphase ^= 1; }
      }
      if (!ok) break;
      if (KSPLIT == 1 && m < g.M) {
        const RowMap rm = map_row(m, g.epi);
        split_epilogue_64<EPI, OUT>(acc, rm, n0, g);
      }
      __syncwarp();
    }
  }

  if constexpr (KSPLIT == 2) {
    // One tile per cluster.  The second pair's sums go to the first pair's CTA of the same rank, 16
    // bytes per lane and store: [epilogue warp][4-column group][lane].
    const int ew = warp - 2;
    const bool epi_warp = warp >= 2 && warp < 2 + Cfg::EPI_WARPS;
    __syncwarp();
    cluster_sync_all();  // every MMA of both pairs is complete: the first pair's ring is idle
    if (part == 1 && epi_warp) {
      const uint32_t dst = map_to_cta(smem_u32(smem), rank) + static_cast<uint32_t>((ew * (CPW / 4) * 32 + lane) * 16);
#pragma unroll
      for (int i = 0; i < CPW / 4; ++i)
        st_cluster_v4(dst + i * 512, acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
    }
    cluster_sync_all();  // release / acquire: the sums are visible to the first pair
    if (part == 0 && epi_warp) {
      const float4* src = reinterpret_cast<const float4*>(smem) + ew * (CPW / 4) * 32 + lane;
#pragma unroll
      for (int i = 0; i < CPW / 4; ++i) {
        const float4 t = src[i * 32];
        acc[4 * i] += t.x; acc[4 * i + 1] += t.y; acc[4 * i + 2] += t.z; acc[4 * i + 3] += t.w;
      }
      const GemmArgs& g = pair < end0 ? p0.g : pair < end1 ? p1.g : p2.g;
      const int lt = pair - (pair < end0 ? 0 : pair < end1 ? end0 : end1);
      const int m = (lt / g.tiles_n) * (2 * S_BM) + static_cast<int>(rank) * S_BM + (warp & 3) * 32 + lane;
      const int n0 = (lt % g.tiles_n) * PBN + (ew >> 2) * CPW;
      if (m < g.M) {
        const RowMap rm = map_row(m, g.epi);
        split_epilogue_64<EPI, OUT>(acc, rm, n0, g);
      }
      __syncwarp();
    }
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*s_abort) drain_after_abort();
  cluster_sync_all();  // no remote arrival or multicast commit may target an exited CTA
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
  }
}

template <int PBN, int EPI, int OUT, int KSPLIT>
int launch_split_inst(const SplitProblem* p, const int* end, cudaStream_t stream) {
  using Cfg = SplitCfg<PBN>;
  auto kern = gemm_split_tcgen05_kernel<PBN, EPI, OUT, KSPLIT>;
  static std::mutex attr_mutex;
  static bool attr_done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (!attr_done[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
      if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(gemm_split)");
      attr_done[dev] = true;
    }
  }
  const int tiles = end[2], most = device_sm_count() / 2;
  launch_dependent(kern, 2 * KSPLIT * (KSPLIT == 2 || tiles < most ? tiles : most), Cfg::THREADS, Cfg::SMEM_BYTES, stream,
                   p[0], p[1], p[2], end[0], end[1], tiles);
  return after_launch("gemm_split_tcgen05_kernel");
}

template <int EPI, int OUT>
int launch_split_width(int bn, int ksplit, const SplitProblem* p, const int* end, cudaStream_t st) {
  if constexpr (EPI == EPI_GATE_RESID) {  // the GEMMs with few tiles and a long K
    if (ksplit == 2)
      return bn == 128 ? launch_split_inst<128, EPI, OUT, 2>(p, end, st) : launch_split_inst<64, EPI, OUT, 2>(p, end, st);
  }
  return bn == 128 ? launch_split_inst<128, EPI, OUT, 1>(p, end, st) : launch_split_inst<64, EPI, OUT, 1>(p, end, st);
}

int validate_split(const SplitGemmProblem& q, int N, int K) {
  const GemmEpilogue& e = q.epi;
  if (!q.A || !q.W || !e.out || q.M <= 0 || N <= 0 || K <= 0 || K % 8 || N % 8 || q.a_plane % 8 || q.w_plane % 8 ||
      (reinterpret_cast<uintptr_t>(q.A) & 15) || (reinterpret_cast<uintptr_t>(q.W) & 15) || e.alpha != 1.0f) {
    set_last_error("gemm_split: invalid argument (M %d N %d K %d)", q.M, N, K);
    return ST_INVALID_ARG;
  }
  const bool planes = e.out_plane > 0;
  if (e.mode != EPI_UNPATCHIFY &&
      ((reinterpret_cast<uintptr_t>(e.out) & 15) || e.ldo % 8 || e.out_plane % 8 || (!planes && !e.out_f32))) {
    set_last_error("gemm_split: output must be fp32 or bf16 planes, 16-byte aligned");
    return ST_INVALID_ARG;
  }
  if (planes && e.mode != EPI_BIAS_GELU && e.mode != EPI_QKV_NORM) {
    set_last_error("gemm_split: no plane output for epilogue mode %d", e.mode);
    return ST_UNSUPPORTED;
  }
  if (e.mode == EPI_QKV_NORM && (e.do_norm && e.qk_cols % 128 != 0)) {
    set_last_error("gemm_split: fused q/k norm needs head_dim 64");
    return ST_INVALID_ARG;
  }
  if (e.mode == EPI_GATE_RESID && (!e.gate || !e.resid || e.gate_stride % 4)) {
    set_last_error("gemm_split: gate/residual epilogue needs gate and resid pointers");
    return ST_INVALID_ARG;
  }
  if (e.mode == EPI_ADD_TABLE && (!e.table || e.rows_in <= 0)) {
    set_last_error("gemm_split: table epilogue needs table and rows_in");
    return ST_INVALID_ARG;
  }
  return ST_OK;
}

int build_split(SplitProblem* pp, const SplitGemmProblem& q, int N, int K, int bn, int* dev_status) {
  GemmArgs& g = pp->g;
  g.M = q.M; g.N = N; g.K = K;
  g.k_blocks = (K + S_KB - 1) / S_KB;
  g.tiles_m = (q.M + 2 * S_BM - 1) / (2 * S_BM);
  g.tiles_n = (N + bn - 1) / bn;
  g.epi = q.epi;
  g.status = dev_status;
  g.tma_store = 0;
  const long esz = q.epi.out_plane > 0 ? 2 : 4;
  g.wide_store = (q.epi.ldo * esz) % 32 == 0 && (q.epi.out_plane * 2) % 32 == 0 &&
                 (reinterpret_cast<uintptr_t>(q.epi.out) & 31) == 0;
  int rc = encode_tmap_3d(&pp->tmA, q.A, 2, K, q.M, 3, static_cast<uint64_t>(K) * 2, q.a_plane * 2, S_KB, S_BM, 3);
  if (rc) return rc;
  return encode_tmap_3d(&pp->tmW, q.W, 2, K, N, 3, static_cast<uint64_t>(K) * 2, q.w_plane * 2, S_KB, bn / 2, 3);
}

// How many clusters of four the device holds at once (a GPC whose SM count is not a multiple of four
// leaves some without work), from the occupancy of the widest instantiation.
long max_clusters_of_four() {
  static std::mutex mu;
  static int known[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (known[dev] == 0) {
    using Cfg = SplitCfg<128>;
    auto kern = gemm_split_tcgen05_kernel<128, EPI_GATE_RESID, 1, 2>;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(4);
    cfg.blockDim = dim3(Cfg::THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known[dev] = n > 0 ? n : -1;
  }
  return known[dev];
}

// The tile width (and, for the gate + residual GEMMs, whether two pairs share a tile's K) with the least
// (waves over the CTA pairs) x (K blocks of a pair) x (time of a block).  In units of 24 cycles a
// block takes 74 at PBN = 128 (measured: 24 MMAs of 64 cycles, a seventh on top) and 56 at PBN = 64 (480
// rows of TMA per CTA); handing the sums over costs two cluster barriers and PBN / 2 KiB of
// distributed shared memory per CTA.
int choose_split_width(long row_tiles, int N, int k_blocks, bool may_split, int* ksplit) {
  const long pairs = device_sm_count() / 2 > 0 ? device_sm_count() / 2 : 1;
  int best = 128;
  long best_cost = 0;
  const int bn[2] = {128, 64}, cost[2] = {74, 56};
  *ksplit = 1;
  for (int i = 0; i < 2; ++i) {
    const long tiles = row_tiles * ((N + bn[i] - 1) / bn[i]);
    const long c = (tiles + pairs - 1) / pairs * cost[i] * k_blocks;
    if (i == 0 || c < best_cost) { best = bn[i]; best_cost = c; *ksplit = 1; }
    if (may_split && k_blocks >= 2 && tiles <= max_clusters_of_four()) {
      const long cs = (k_blocks + 1) / 2 * cost[i] + 125 + 2 * bn[i] / 3;
      if (cs < best_cost) { best = bn[i]; best_cost = cs; *ksplit = 2; }
    }
  }
  return best;
}

}  // namespace

int launch_gemm_split(const SplitGemmProblem* q, int n, int N, int K, int* dev_status, cudaStream_t stream) {
  if (n < 1 || n > 3) {
    set_last_error("gemm_split: one to three problems (got %d)", n);
    return ST_INVALID_ARG;
  }
  const SplitGemmProblem& a = q[0];
  long row_tiles = 0;
  for (int i = 0; i < n; ++i) {
    int rc = validate_split(q[i], N, K);
    if (rc) return rc;
    if (q[i].epi.mode != a.epi.mode || (q[i].epi.out_plane > 0) != (a.epi.out_plane > 0) ||
        q[i].epi.out_f32 != a.epi.out_f32) {
      set_last_error("gemm_split: grouped problems need the same epilogue kind");
      return ST_INVALID_ARG;
    }
    row_tiles += (q[i].M + 2 * S_BM - 1) / (2 * S_BM);
  }
  int ksplit = 1;
  const int bn = choose_split_width(row_tiles, N, (K + S_KB - 1) / S_KB, a.epi.mode == EPI_GATE_RESID, &ksplit);
  SplitProblem p[3];
  int end[3] = {0, 0, 0}, tiles = 0;
  for (int i = 0; i < 3; ++i) {
    if (i < n) {
      int rc = build_split(&p[i], q[i], N, K, bn, dev_status);
      if (rc) return rc;
      tiles += p[i].g.tiles_m * p[i].g.tiles_n;
    } else {
      p[i] = p[0];  // no tiles
    }
    end[i] = tiles;
  }
  const bool planes = a.epi.out_plane > 0;
  switch (a.epi.mode) {
    case EPI_BIAS: return launch_split_width<EPI_BIAS, 1>(bn, ksplit, p, end, stream);
    case EPI_BIAS_GELU:
      if (planes) return launch_split_width<EPI_BIAS_GELU, 2>(bn, ksplit, p, end, stream);
      break;
    case EPI_QKV_NORM:
      return planes ? launch_split_width<EPI_QKV_NORM, 2>(bn, ksplit, p, end, stream)
                    : launch_split_width<EPI_QKV_NORM, 1>(bn, ksplit, p, end, stream);
    case EPI_GATE_RESID: return launch_split_width<EPI_GATE_RESID, 1>(bn, ksplit, p, end, stream);
    case EPI_ADD_TABLE: return launch_split_width<EPI_ADD_TABLE, 1>(bn, ksplit, p, end, stream);
    case EPI_UNPATCHIFY:
      return a.epi.out_f32 ? launch_split_width<EPI_UNPATCHIFY, 1>(bn, ksplit, p, end, stream)
                           : launch_split_width<EPI_UNPATCHIFY, 0>(bn, ksplit, p, end, stream);
    default: break;
  }
  set_last_error("gemm_split: unsupported epilogue mode %d", a.epi.mode);
  return ST_UNSUPPORTED;
}

}  // namespace sd3
