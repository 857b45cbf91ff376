// CTA-pair variant of the tcgen05 GEMM: two CTAs (a cluster of two on
// neighbouring SMs) cooperate on 256 x 256 output tiles (256 x 128 or, for gate + residual, 256 x 64 where those fill
// the SMs better: launch_rules.h) with tcgen05.mma.cta_group::2.  One launch can carry up to THREE problems of the same
// shape class (same N, K and epilogue: the image-stream GEMM of a block, its
// small context-stream twin and, for QKV, the second projection of a dual block);
// the persistent tile loop runs one problem's tiles after the other's, so the small
// ones ride in the tail of the large one instead of being launches of their own
// that fill less than a wave (the third problem: forward of one 256x256 image 3284 -> 3133 us, 512x512
// 4467 -> 4407 us, 1024x1024 unchanged).  A dual block's two out-projections add to the same rows: a pair that has run
// a tile of the first runs the third problem's tile of the same place next (pair_tiles.h; against a launch of their own,
// 256x256 2335 -> 2311 us, 512x512 3719 -> 3690, 1024x1024 unchanged).
//
//   acc[m, n] = sum_k A[m, k] * W[n, k]        A: (M, K) K-major, W: (N, K) K-major
//
// Per 64-wide K block each CTA loads only its own 128 rows of A and its own
// 128-row half of the W tile (32 KiB instead of the 48 KiB a lone CTA needs
// for a 128 x 256 tile); the tensor cores of both SMs read the two W halves
// from both shared memories.  That cuts the L2 -> shared-memory traffic per
// FLOP by a third and leaves room for a six-stage ring.  One warp of the even CTA of the
// pair issues all MMAs, one warp of each CTA its loads.  Both stay converged and an elected lane issues:
// descriptors and addresses then live in uniform registers.  From a branch taken by lane 0 alone an MMA took
// 63-88 cycles to issue (a 128-wide MMA runs 64) and a slot's loads 740; elected, 33-39 and under 300.
// Measured, lane 0 with two issuing threads that took turns -> elected lane of one warp (us, weights from
// HBM): N = 1536, K = 6144, 589 rows 26.9 -> 20.0, 4429 rows 72.6 -> 68.8; QKV 4429 rows 60.9 -> 49.1, 13287 rows
// 143 -> 123 (147 -> 130 on another GPU); GELU 4429 rows 68.3 -> 61.9.  Completion is signalled to both CTAs with
// tcgen05.commit ... multicast::cluster.  Each CTA keeps the accumulator rows
// of its own half of M in its own TMEM (two buffers of 256 columns) and drains
// them through the same fused epilogues as the one-CTA kernel.
//
// Loads are plain tiled TMA (cta_group::2 form so the peer's transaction bytes
// can be credited to the leader's barrier); nothing here is a multicast load.
#include <cuda.h>
#include <mutex>

#include "gemm_epilogue.cuh"
#include "kernels.h"
#include "launch_rules.h"
#include "pair_tiles.h"
#include "ptx.cuh"

namespace sd3 {

int encode_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t inner,
                   uint64_t outer, uint64_t ld_bytes, uint32_t box_inner, uint32_t box_outer);
int device_sm_count();

namespace {

using namespace gemm_detail;

constexpr int P_BM = 128;            // rows of A per CTA (256 per pair)
constexpr int P_KBYTES = 128;        // bytes of K per stage row (64 bf16)
constexpr int P_A_BYTES = P_BM * P_KBYTES;
// PBN = output columns per pair tile (256, 128 or 64); each CTA loads PBN / 2 rows of W
__host__ __device__ constexpr int pair_b_bytes(int pbn) { return (pbn / 2) * P_KBYTES; }
__host__ __device__ constexpr int pair_stage_bytes(int pbn) { return P_A_BYTES + pair_b_bytes(pbn); }  // 32 / 24 / 20 KiB
// The epilogues that leave through shared memory (TMA reduction or TMA store) get 4 KiB per
// epilogue warp.
constexpr int P_RED_BYTES = 4096;
__host__ __device__ constexpr bool pair_stages_out(int epi, bool out_f32) {
  return epi == EPI_GATE_RESID || (!out_f32 && (epi == EPI_BIAS || epi == EPI_BIAS_GELU || epi == EPI_QKV_NORM));
}
// Six stages of 32 KiB (eight of 24 KiB), handed over in slots of one (two): a full and an empty barrier, one
// wait and one commit each.  A stage of the wide tile is 512 cycles of MMA and single hand-overs refill the
// ring sooner (N = 1536, K = 6144, 4429 rows: 69.1 us against 70.9 with slots of two; 13287 rows: 191 against 207);
// one of the narrow tile is 256 cycles, less than a hand-over takes (589 rows: 24.6 us, with slots of two 20.4).
__host__ __device__ constexpr int pair_stages(int pbn) { return pbn == 256 ? 6 : 8; }
__host__ __device__ constexpr int pair_slot(int pbn) { return pbn == 256 ? 1 : 2; }
__host__ __device__ constexpr int pair_red_bytes(int epi, bool out_f32) {
  return pair_stages_out(epi, out_f32) ? EPI_WARPS * P_RED_BYTES : 0;
}
constexpr int P_THREADS = 64 + 32 * EPI_WARPS;
__host__ __device__ constexpr int pair_smem_bytes(int epi, bool out_f32, int pbn) {
  return pair_stages(pbn) * pair_stage_bytes(pbn) + pair_red_bytes(epi, out_f32) + 256 + 1024;
}

// One problem of a (possibly grouped) launch
struct PairProblem {
  CUtensorMap tmA, tmW, tmR;  // tmR: fp32 residual (gate + residual) or bf16 output (TMA store)
  GemmArgs g;
};

template <int EPI, bool OUT_F32, bool FP8, int PBN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_pair_tcgen05_kernel(const __grid_constant__ PairProblem p0, const __grid_constant__ PairProblem p1,
                         const __grid_constant__ PairProblem p2, const PairTiles all) {
  // M = 256 across the pair; operands bf16, or e4m3 (128 K-elements per 128-byte stage row,
  // 32 per instruction: the byte arithmetic of the stages is the same)
  constexpr uint32_t IDESC = FP8 ? make_idesc(0, 0, 2 * P_BM, PBN, 0, 0) : make_idesc(1, 1, 2 * P_BM, PBN, 0, 0);
  constexpr int P_BN_HALF = PBN / 2;
  constexpr int P_STAGE_BYTES = pair_stage_bytes(PBN);
  constexpr int P_TMEM_COLS = 2 * PBN;  // two accumulators

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  constexpr int P_STAGES = pair_stages(PBN);
  static_assert(EPI_WARPS * ((PBN + 63) / 64) * P_RED_BYTES <= P_STAGES * P_STAGE_BYTES, "the last tile's boxes fit the ring");
  uint8_t* red_smem = smem + P_STAGES * P_STAGE_BYTES;  // 1024-byte aligned: stages are 32 / 24 / 20 KiB each
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + P_STAGES * P_STAGE_BYTES + pair_red_bytes(EPI, OUT_F32));
  uint64_t* empty_bar = full_bar + P_STAGES;
  uint64_t* tfull_bar = empty_bar + P_STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // known uniform
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  // tiles of 256 x PBN
  const PairTiles tiles{all.end0, all.end1, all.end2, EPI == EPI_GATE_RESID ? all.sum : 0};
  const int end0 = tiles.end0, end1 = tiles.end1, num_tiles = tiles.end2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);   // leader's expect_tx arrival; bytes of both CTAs
      mbar_init(&empty_bar[s], 1);  // one multicast commit per use
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * EPI_WARPS);  // epilogue warps of both CTAs (leader's copy is used)
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
    tmem_alloc_pair(tmem_slot, P_TMEM_COLS);
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

  constexpr int SLOT = pair_slot(PBN);
  constexpr int NSLOT = P_STAGES / SLOT;
  const int KB = p0.g.k_blocks;  // the same K for all problems

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs, one warp) --------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const bool issuer = elect_one();
    constexpr int KEL = FP8 ? P_KBYTES : P_KBYTES / 2;  // K elements per stage
    const uint32_t ring = smem_u32(smem);
    const uint32_t full_local = smem_u32(full_bar), full_leader = map_to_cta(full_local, 0);
    // stages [kb, kb + SLOT) of a tile into slot st; all bytes of the slot (both CTAs) are credited to the
    // leader's barrier
    auto load_w = [&](const CUtensorMap* tmW, int st, int kb, int n0) {
      if (rank == 0) mbar_expect_tx_at(full_local + 8 * st, min(SLOT, KB - kb) * (2 * P_STAGE_BYTES));
#pragma unroll
      for (int i = 0; i < SLOT; ++i)
        if (SLOT == 1 || kb + i < KB)
          tma_load_2d_pair_at(ring + (st * SLOT + i) * P_STAGE_BYTES + P_A_BYTES, tmW, full_leader + 8 * st,
                              (kb + i) * KEL, n0);
    };
    auto load_a = [&](const CUtensorMap* tmA, int st, int kb, int m0) {
#pragma unroll
      for (int i = 0; i < SLOT; ++i)
        if (SLOT == 1 || kb + i < KB)
          tma_load_2d_pair_at(ring + (st * SLOT + i) * P_STAGE_BYTES, tmA, full_leader + 8 * st, (kb + i) * KEL, m0);
    };
    int pre = 0;  // slots of the first tile whose weights are under way before the wait
    bool waited = false;
    for (int tile = pair; tile < num_tiles && ok; tile = tiles.next(tile, num_pairs)) {
      const PairProblem& pp = tile < end0 ? p0 : tile < end1 ? p1 : p2;
      const int lt = tile - (tile < end0 ? 0 : tile < end1 ? end0 : end1);
      const int m0 = (lt / pp.g.tiles_n) * (2 * P_BM) + static_cast<int>(rank) * P_BM;
      const int n0 = (lt % pp.g.tiles_n) * PBN + static_cast<int>(rank) * P_BN_HALF;
      const CUtensorMap *tmA = &pp.tmA, *tmW = &pp.tmW;
      if (!waited) {
        if (p0.g.epi.w_static)
          for (; pre < NSLOT && pre * SLOT < KB; ++pre)
            if (issuer) load_w(tmW, pre, pre * SLOT, n0);
        grid_dep_wait();
        waited = true;
      }
      for (int kb = 0; kb < KB; kb += SLOT) {
        if (pre > 0) {
          --pre;
        } else {
          if (!mbar_wait_all(&empty_bar[stage], phase ^ 1, wc, DEV_TIMEOUT_EMPTY)) { ok = false; break; }
          if (issuer) load_w(tmW, stage, kb, n0);
        }
        if (issuer) load_a(tmA, stage, kb, m0);
        if (++stage == NSLOT) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader only, one warp) --------
    if (rank == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      const bool issuer = elect_one();
      const uint64_t desc0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
      for (int tile = pair; tile < num_tiles && ok; tile = tiles.next(tile, num_pairs)) {
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * PBN);
        if (!mbar_wait_all(&tempty_bar[acc], acc_phase ^ 1, wc, DEV_TIMEOUT_TMEM_EMPTY)) break;
        for (int kb = 0; kb < KB; kb += SLOT) {
          if (!mbar_wait_all(&full_bar[stage], phase, wc, DEV_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after_sync();
          if (issuer) {
#pragma unroll
            for (int i = 0; i < SLOT; ++i) {
              if (SLOT > 1 && kb + i >= KB) break;
              const uint64_t a_desc = desc0 + static_cast<uint32_t>((stage * SLOT + i) * (P_STAGE_BYTES >> 4));
              const uint64_t b_desc = a_desc + (P_A_BYTES >> 4);
#pragma unroll
              for (int k = 0; k < P_KBYTES / 32; ++k) {
                const uint64_t adv = static_cast<uint64_t>((k * 32) >> 4);
                if constexpr (FP8)
                  mma_f8_ss_pair(d_tmem, a_desc + adv, b_desc + adv, IDESC, (kb | i | k) != 0);
                else
                  mma_f16_ss_pair(d_tmem, a_desc + adv, b_desc + adv, IDESC, (kb | i | k) != 0);
              }
            }
            mma_commit_pair(&empty_bar[stage], 3);                     // frees the slot in both CTAs
            if (kb + SLOT >= KB) mma_commit_pair(&tfull_bar[acc], 3);  // accumulator ready in both CTAs
          }
          if (++stage == NSLOT) { stage = 0; phase ^= 1; }
        }
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ----------------------
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < num_tiles; tile = tiles.next(tile, num_pairs)) {
      const PairProblem& pp = tile < end0 ? p0 : tile < end1 ? p1 : p2;
      const GemmArgs& g = pp.g;
      const int lt = tile - (tile < end0 ? 0 : tile < end1 ? end0 : end1);
      const int m0 = (lt / g.tiles_n) * (2 * P_BM) + static_cast<int>(rank) * P_BM;
      const int n0 = (lt % g.tiles_n) * PBN;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) +
                             static_cast<uint32_t>(acc * PBN);
      bool drained;
      // After the pair's last tile the operand ring is idle (its accumulator is complete, so every load has landed
      // and every MMA has read it): each box of the epilogue gets a buffer of its own there, and none waits for the
      // one before it to have been read.  us of a launch, before -> after: gate + residual K 1536, 589 rows 8.8 -> 8.2,
      // 1357 rows 9.6 -> 9.3; K 6144, 589 rows 20.3 -> 19.7; GELU 1357 rows 23.5 -> 22.5, 4429 rows 61.1 -> 59.2.  (256-wide
      // QKV tiles lose it to spilled registers: 4429 rows 47.4 -> 50.5.)
      constexpr bool OWN_BOXES = !(EPI == EPI_QKV_NORM && PBN == 256);
      const bool last = OWN_BOXES && tiles.next(tile, num_pairs) >= num_tiles;
      constexpr int BOXES = PBN / 2 / (EPI == EPI_GATE_RESID ? 32 : 64);  // of a warp and tile
      uint8_t* box = last ? smem + (warp - 2) * (BOXES * P_RED_BYTES) : red_smem + (warp - 2) * P_RED_BYTES;
      const int box_step = last ? P_RED_BYTES : 0;
      if constexpr (EPI == EPI_GATE_RESID)
        drained = drain_tile_gate_reduce<PBN>(t_row, m0 + quad * 32, n0, half, g, &pp.tmR, &tfull_bar[acc],
                                              acc_phase, wc, box, box_step, tiles.sum && tile >= end1);
      else
        drained = drain_tile<PBN, EPI, OUT_F32>(t_row, m0 + row, n0, half, g, &tfull_bar[acc], acc_phase, wc,
                                                (pair_stages_out(EPI, OUT_F32) && g.tma_store) ? box : nullptr,
                                                &pp.tmR, box_step);
      if (!drained) break;
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[acc]), 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if constexpr (pair_stages_out(EPI, OUT_F32)) {
      if (lane == 0) bulk_wait_group0();  // every reduction / store of this warp has landed
    }
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*s_abort) drain_after_abort();
  cluster_sync_all();  // no remote arrival or multicast commit may target an exited CTA
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, P_TMEM_COLS);
  }
}

template <int EPI, bool OUT_F32, bool FP8, int PBN>
int launch_pair_inst(const PairProblem* p, const PairTiles& tiles, cudaStream_t stream) {
  auto kern = gemm_pair_tcgen05_kernel<EPI, OUT_F32, FP8, PBN>;
  constexpr int SMEM = pair_smem_bytes(EPI, OUT_F32, PBN);
  static std::mutex attr_mutex;
  static bool attr_done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (!attr_done[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
      if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(gemm_pair)");
      attr_done[dev] = true;
    }
  }
  const int max_pairs = device_sm_count() / 2;
  const int pairs = tiles.starts() < max_pairs ? tiles.starts() : max_pairs;
  launch_dependent(kern, 2 * pairs, P_THREADS, SMEM, stream, p[0], p[1], p[2], tiles);
  return after_launch("gemm_pair_tcgen05_kernel");
}

// the epilogues that a forward uses exist for both tile widths, the others for 256 only
template <int EPI, bool OUT_F32, bool FP8>
int launch_pair_width(int pbn, const PairProblem* p, const PairTiles& tiles, cudaStream_t stream) {
  constexpr bool narrow_built = (OUT_F32 && (EPI == EPI_GATE_RESID || EPI == EPI_BIAS || EPI == EPI_ADD_TABLE)) ||
                                (!OUT_F32 && (EPI == EPI_BIAS || EPI == EPI_BIAS_GELU || EPI == EPI_QKV_NORM));
  if constexpr (narrow_built) {
    if (pbn == 128) return launch_pair_inst<EPI, OUT_F32, FP8, 128>(p, tiles, stream);
  }
  if constexpr (EPI == EPI_GATE_RESID) {
    if (pbn == 64) return launch_pair_inst<EPI, OUT_F32, FP8, 64>(p, tiles, stream);
  }
  return launch_pair_inst<EPI, OUT_F32, FP8, 256>(p, tiles, stream);
}

bool narrow_tiles_built(const GemmEpilogue& epi) {
  if (epi.out_f32) return epi.mode == EPI_GATE_RESID || epi.mode == EPI_BIAS || epi.mode == EPI_ADD_TABLE;
  return epi.mode == EPI_BIAS || epi.mode == EPI_BIAS_GELU || epi.mode == EPI_QKV_NORM;
}

// Tensor maps and arguments of one problem for pair tiles of width pbn.
int build_problem(PairProblem* pp, const GemmProblem& q, int operand_dtype, int N, int K, int pbn,
                  int* dev_status) {
  const bool fp8 = operand_dtype == OPERAND_E4M3;
  const int eb = fp8 ? 1 : 2, kel = P_KBYTES / eb;  // element bytes, K elements per stage
  const GemmEpilogue& epi = q.epi;
  const int M = q.M;
  GemmArgs& g = pp->g;
  g.M = M; g.N = N; g.K = K;
  g.k_blocks = (K + kel - 1) / kel;
  g.tiles_m = (M + 2 * P_BM - 1) / (2 * P_BM);
  g.tiles_n = N / pbn;
  g.epi = epi;
  g.status = dev_status;
  {
    const long esz = epi.out_f32 ? 4 : 2;
    g.wide_store = (N % 16 == 0) && ((epi.ldo * esz) % 32 == 0) &&
                   ((reinterpret_cast<uintptr_t>(epi.out) & 31) == 0);
  }
  int rc = encode_tmap_2d(&pp->tmA, q.A, eb, (uint64_t)K, (uint64_t)M, (uint64_t)q.lda * eb, kel, P_BM);
  if (rc) return rc;
  rc = encode_tmap_2d(&pp->tmW, q.W, eb, (uint64_t)K, (uint64_t)N, (uint64_t)q.ldw * eb, kel, pbn / 2);
  if (rc) return rc;
  const bool f32 = epi.out_f32 != 0;
  pp->tmR = pp->tmA;  // placeholder for the epilogues that neither reduce nor store through TMA
  if (epi.mode == EPI_GATE_RESID) {
    if (epi.out != epi.resid) {
      set_last_error("gemm_pair: gate/residual epilogue updates the residual in place (out must equal resid)");
      return ST_INVALID_ARG;
    }
    rc = encode_tmap_2d(&pp->tmR, epi.resid, 4, (uint64_t)N, (uint64_t)M, (uint64_t)epi.ldo * 4, 32, 32);
    if (rc) return rc;
  }
  // bf16 outputs leave through a TMA store when every warp's 32 rows are 32 consecutive
  // output rows that all exist
  g.tma_store = 0;
  if (!f32 && !epi.out_e4m3 && M % 32 == 0 && (epi.rows_in == 0 || epi.rows_in % 32 == 0) &&
      (epi.mode == EPI_BIAS || epi.mode == EPI_BIAS_GELU || epi.mode == EPI_QKV_NORM) && epi.hg_groups <= 1 &&
      (epi.ldo * 2) % 16 == 0 && (reinterpret_cast<uintptr_t>(epi.out) & 15) == 0) {
    // with a row remap the last sample's rows end at (samples - 1) * rows_out + row_off + rows_in
    const uint64_t extent = epi.rows_in > 0
                                ? (uint64_t)(M / epi.rows_in - 1) * epi.rows_out + epi.row_off + epi.rows_in
                                : (uint64_t)M;
    rc = encode_tmap_2d(&pp->tmR, epi.out, 2, (uint64_t)N, extent, (uint64_t)epi.ldo * 2, 64, 32);
    if (rc) return rc;
    g.tma_store = 1;
  }
  return ST_OK;
}

}  // namespace

// Whether the CTA-pair kernel covers this problem (N a multiple of 256, enough rows to fill
// pair tiles, an epilogue that is instantiated for the operand type).
bool gemm_pair_supported(int operand_dtype, int M, int N, int K, const GemmEpilogue& epi) {
  (void)K;
  if (N % 256 != 0 || M < 2 * P_BM) return false;
  if (epi.mode == EPI_UNPATCHIFY) return false;
  if (operand_dtype == OPERAND_E4M3) {
    // e4m3 instantiations exist for the epilogues of the block GEMMs
    if (epi.mode == EPI_GATE_RESID) return epi.out_f32 != 0;
    return (epi.mode == EPI_QKV_NORM || epi.mode == EPI_BIAS_GELU || epi.mode == EPI_BIAS) && !epi.out_f32;
  }
  return operand_dtype == OPERAND_BF16;
}

// One to three problems of the same N, K, operand type and epilogue kind.
int launch_gemm_pair(const GemmProblem* q, int n, int operand_dtype, int N, int K, int* dev_status,
                     cudaStream_t stream) {
  const bool fp8 = operand_dtype == OPERAND_E4M3;
  const GemmProblem& a = q[0];
  // by itself such a problem is an ordinary one: it comes after the first in stream order
  const bool sum = n > 1 && q[n - 1].epi.adds_after;
  long tiles256 = 0;
  for (int i = 0; i < n; ++i) {
    if (n > 1 && q[i].epi.adds_after &&
        (i != n - 1 || a.epi.mode != EPI_GATE_RESID || q[i].M != a.M || q[i].epi.resid != a.epi.resid ||
         q[i].epi.ldo != a.epi.ldo)) {
      set_last_error("gemm_pair: a problem that adds after the first has its rows and its residual, and comes last");
      return ST_INVALID_ARG;
    }
    if (q[i].epi.mode != a.epi.mode || q[i].epi.out_f32 != a.epi.out_f32) {
      set_last_error("gemm_pair: grouped problems need the same epilogue kind");
      return ST_INVALID_ARG;
    }
    tiles256 += static_cast<long>((q[i].M + 255) / 256) * (N / 256);
  }
  const long after256 = sum ? static_cast<long>((a.M + 255) / 256) * (N / 256) : 0;
  const int pbn = !narrow_tiles_built(a.epi) ? 256
                                             : pair_tile_width(tiles256, after256, K, fp8, a.epi.mode == EPI_GATE_RESID,
                                                               device_sm_count() / 2);
  PairProblem p[3];
  int end[3] = {0, 0, 0}, count = 0;
  for (int i = 0; i < 3; ++i) {
    const int j = sum && i == 2 ? n - 1 : i < (sum ? n - 1 : n) ? i : -1;  // one that adds after the first is the third
    if (j >= 0) {
      int rc = build_problem(&p[i], q[j], operand_dtype, N, K, pbn, dev_status);
      if (rc) return rc;
      count += p[i].g.tiles_m * p[i].g.tiles_n;
    } else {
      p[i] = p[0];  // no tiles
    }
    end[i] = count;
  }
  const PairTiles tiles{end[0], end[1], end[2], sum ? 1 : 0};
  const bool f32 = a.epi.out_f32 != 0;
  if (fp8) {
    switch (a.epi.mode) {
      case EPI_BIAS: return launch_pair_width<EPI_BIAS, false, true>(pbn, p, tiles, stream);
      case EPI_BIAS_GELU: return launch_pair_width<EPI_BIAS_GELU, false, true>(pbn, p, tiles, stream);
      case EPI_QKV_NORM: return launch_pair_width<EPI_QKV_NORM, false, true>(pbn, p, tiles, stream);
      case EPI_GATE_RESID: return launch_pair_width<EPI_GATE_RESID, true, true>(pbn, p, tiles, stream);
      default: break;
    }
    set_last_error("gemm_pair: no e4m3 instantiation for epilogue mode %d", a.epi.mode);
    return ST_UNSUPPORTED;
  }
  switch (a.epi.mode) {
    case EPI_BIAS:
      return f32 ? launch_pair_width<EPI_BIAS, true, false>(pbn, p, tiles, stream)
                 : launch_pair_width<EPI_BIAS, false, false>(pbn, p, tiles, stream);
    case EPI_BIAS_GELU:
      return f32 ? launch_pair_width<EPI_BIAS_GELU, true, false>(pbn, p, tiles, stream)
                 : launch_pair_width<EPI_BIAS_GELU, false, false>(pbn, p, tiles, stream);
    case EPI_GATE_RESID:
      if (!f32) break;
      return launch_pair_width<EPI_GATE_RESID, true, false>(pbn, p, tiles, stream);
    case EPI_QKV_NORM:
      return f32 ? launch_pair_width<EPI_QKV_NORM, true, false>(pbn, p, tiles, stream)
                 : launch_pair_width<EPI_QKV_NORM, false, false>(pbn, p, tiles, stream);
    case EPI_ADD_TABLE:
      if (!f32) break;
      return launch_pair_width<EPI_ADD_TABLE, true, false>(pbn, p, tiles, stream);
    default:
      break;
  }
  set_last_error("gemm_pair: unsupported epilogue mode %d / out_f32 %d", a.epi.mode, a.epi.out_f32);
  return ST_UNSUPPORTED;
}

}  // namespace sd3
