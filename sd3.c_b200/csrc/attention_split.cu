// fp32 attention for head_dim 64 on tcgen05 / TMEM: q, k, v and the
// probabilities are three bf16 planes each (x = h + m + l exactly, split3.cuh),
// every product is formed by the six plane products above 2^-25, softmax
// statistics, exponentials and the running output are fp32.
//
// One CTA owns 128 queries of one (sample, head).  Warp 0 streams the planes of
// K (two 128-key stages) and V (two 64-key halves) with TMA; an elected lane of
// warp 1 issues the MMAs; eight softmax warps own half the keys of a query row
// per thread (TMEM lane == row).  Per 128 keys:
//   S = Q K^T   24 MMAs of N = 128, smallest products first;
//   P           = 2^(S c - m c) in registers, split and written to TMEM planes;
//   acc = P V   three MMAs per 16 keys: Ph x [Vh Vm Vl] (N = 192), Pm x [Vh Vm]
//               (N = 128), Pl x [Vh] (N = 64) into three column blocks that hold
//               the products of size 1, 2^-8 and 2^-16 (V's planes lie side by
//               side along N; an MMA below N = 128 is issue-bound, so six
//               MMAs of N = 64 would take 300 cycles where these take 210);
//   O = (O + acc) 2^((m_old - m_new) c) in registers, round to nearest: the tensor core's own
//               accumulation truncates and is only used within one tile.
// The score buffer is emptied into registers at once, so the scores of tile j + 1
// run under the exponentials of tile j, and the exponentials and splits of tile
// j + 1 under the products of tile j; what stands between two tiles' products is
// the addition of acc and the store of P.
// Two warps share a row (keys 0..63 and 64..127 of a tile, 32 of the 64 output
// columns each; they exchange the tile's maximum through shared memory): one warp
// per scheduler with a whole row in registers ran 2500 unrolled instructions a
// tile, more than the instruction cache holds, at 0.3 instructions per cycle (8500 cycles a tile).
// What bounds it: the chain scores -> exponentials -> products of a tile, of which the MMAs (1536 + 1680 cycles
// per 128 x 128 tile pair) are about half: tensor pipe 43 %, issue slots 34 %, fixed latencies and polls first
// among the stalls (1024 + 333 tokens).
//
// Measured against attention_simt_kernel (one warp per query, uncoalesced key rows), which this
// replaces for fp32 models with head_dim 64: one dual block of 256 + 77 tokens 2.79 -> 0.49 ms, the
// 24-block model at 512 x 512 668 -> 19.1 ms; the second warp per row: 17.53 -> 16.79 ms.  Error of
// that block's branches against float64: 3.4e-7 (FFMA GEMMs and SIMT attention: 1.6e-6).
#include <cuda.h>
#include <mutex>

#include "kernels.h"
#include "ptx.cuh"
#include "split3.cuh"

namespace sd3 {

int encode_tmap_3d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t d0, uint64_t d1, uint64_t d2,
                   uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t box0, uint32_t box1, uint32_t box2);

namespace {

constexpr int AS_BM = 128, AS_BN = 128, AS_D = 64;
constexpr int AS_PLANE = AS_BN * AS_D * 2;   // 16 KiB: one plane of 128 rows
constexpr int AS_HPLANE = AS_PLANE / 2;      // one plane of 64 rows
constexpr int AS_TILE = 3 * AS_PLANE;        // Q, one K stage, both V halves
constexpr int AS_THREADS = 64 + 8 * 32;
constexpr int AS_S_COL = 0;    // scores: 128 fp32 columns
constexpr int AS_P_COL = 128;  // P: three planes of 64 columns (bf16 pairs)
constexpr int AS_O_COL = 320;  // P V of one tile: three blocks of 64 fp32 columns
constexpr int AS_XCHG_BYTES = 2 * 2 * AS_BM * 4;  // row maxima: [tile parity][half][row]
constexpr int AS_SMEM_BYTES = 4 * AS_TILE + AS_XCHG_BYTES + 256 + 1024;  // Q, two K stages, V

struct SplitAttnArgs {
  int B, T, NH, Tc, E;
  int b0;       // sample of blockIdx.z == 0 (grids hold at most 65535 samples)
  bf16* out_c;  // three planes of B * Tc * E, or null
  bf16* out_x;  // three planes of B * (T - Tc) * E
  float c;      // softmax scale * log2(e)
  int* status;
};

__device__ __forceinline__ float ex2_f32(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));  // without ftz three more instructions
  return y;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__global__ void __launch_bounds__(AS_THREADS, 1)
attention_split_tcgen05_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
                               const __grid_constant__ SplitAttnArgs a0, const __grid_constant__ SplitAttnArgs a1,
                               const int grid0) {
  // grid.x: the query tiles of the first attention, then those of the second (the image-only one of a dual block)
  const bool second = static_cast<int>(blockIdx.x) >= grid0;
  const CUtensorMap& tm = second ? tm1 : tm0;
  const SplitAttnArgs& a = second ? a1 : a0;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* q_smem = smem;                 // [plane][128 rows][128 B]
  uint8_t* k_smem = smem + AS_TILE;       // [stage][plane][128 rows][128 B]
  uint8_t* v_smem = smem + 3 * AS_TILE;   // [half][plane][64 rows][128 B]
  float* s_max = reinterpret_cast<float*>(smem + 4 * AS_TILE);
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + 4 * AS_TILE + AS_XCHG_BYTES);
  uint64_t* k_full = q_full + 1;    // 2
  uint64_t* k_empty = k_full + 2;   // 2
  uint64_t* v_full = k_empty + 2;   // 2
  uint64_t* v_empty = v_full + 2;   // 2
  uint64_t* s_full = v_empty + 2;   // scores of a tile complete
  uint64_t* s_free = s_full + 1;    // scores are in registers (8 arrivals)
  uint64_t* p_ready = s_free + 1;   // P of a tile is in TMEM and acc has been read (8 arrivals)
  uint64_t* pv_done = p_ready + 1;  // products of a tile complete
  uint64_t* xchg = pv_done + 1;     // 4: both warps of a row quadrant have written their maxima
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xchg + 4);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // known uniform
  const int lane = threadIdx.x & 31;
  const int q0 = (static_cast<int>(blockIdx.x) - (second ? grid0 : 0)) * AS_BM, h = blockIdx.y, b = a.b0 + blockIdx.z;
  const int T = a.T, nkv = (T + AS_BN - 1) / AS_BN;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_free, 8);
    mbar_init(p_ready, 8);
    mbar_init(pv_done, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&xchg[i], 2);
    *s_abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tm);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  grid_dep_wait();
  grid_dep_launch();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const WaitCtx wc{s_abort, a.status};

  if (warp == 0) {
    // ------------------------------ TMA producer (a converged warp, one lane issues) ------
    const bool issuer = elect_one();
    // 64 rows from `row` of every plane (plane p of sample b is slab p * B + b); plane_bytes apart
    auto load_rows = [&](uint8_t* dst, int plane_bytes, uint64_t* bar, int col, int row) {
#pragma unroll
      for (int p = 0; p < 3; ++p) tma_load_3d(dst + p * plane_bytes, &tm, bar, col, row, p * a.B + b);
    };
    auto load_k = [&](int j) {
      const int st = j & 1;
      if (j >= 2 && !mbar_wait_all(&k_empty[st], ((j >> 1) - 1) & 1, wc, DEV_TIMEOUT_ATTN_KV)) return false;
      if (issuer) {
        mbar_expect_tx(&k_full[st], AS_TILE);
        uint8_t* d = k_smem + st * AS_TILE;
        load_rows(d, AS_PLANE, &k_full[st], a.E + h * AS_D, j * AS_BN);
        load_rows(d + AS_HPLANE, AS_PLANE, &k_full[st], a.E + h * AS_D, j * AS_BN + 64);
      }
      return true;
    };
    if (issuer) {
      mbar_expect_tx(q_full, AS_TILE);
      load_rows(q_smem, AS_PLANE, q_full, h * AS_D, q0);
      load_rows(q_smem + AS_HPLANE, AS_PLANE, q_full, h * AS_D, q0 + 64);
    }
    bool ok = load_k(0);
    for (int j = 0; j < nkv && ok; ++j) {
      if (j + 1 < nkv) ok = load_k(j + 1);
      for (int hf = 0; hf < 2 && ok; ++hf) {
        if (j >= 1 && !mbar_wait_all(&v_empty[hf], (j - 1) & 1, wc, DEV_TIMEOUT_ATTN_KV)) { ok = false; break; }
        if (issuer) {
          mbar_expect_tx(&v_full[hf], AS_TILE / 2);
          load_rows(v_smem + hf * (AS_TILE / 2), AS_HPLANE, &v_full[hf], 2 * a.E + h * AS_D, j * AS_BN + 64 * hf);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (a converged warp, one lane issues) ------
    constexpr uint32_t IDESC_S = make_idesc(1, 1, AS_BM, AS_BN, 0, 0);
    constexpr uint32_t IDESC_O3 = make_idesc(1, 1, AS_BM, 192, 0, 1);  // V is MN-major
    constexpr uint32_t IDESC_O2 = make_idesc(1, 1, AS_BM, 128, 0, 1);
    constexpr uint32_t IDESC_O1 = make_idesc(1, 1, AS_BM, 64, 0, 1);
    constexpr uint64_t PL = AS_PLANE >> 4;
    constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};  // smallest products first
    const uint32_t s_tmem = tmem_base + AS_S_COL, p_tmem = tmem_base + AS_P_COL, o_tmem = tmem_base + AS_O_COL;
    const uint64_t q_desc = make_smem_desc_sw128(smem_u32(q_smem), 16, 1024);
    const uint64_t k_desc0 = make_smem_desc_sw128(smem_u32(k_smem), 16, 1024);
    // planes 8 KiB apart along N (leading-dimension offset)
    const uint64_t v_desc0 = make_smem_desc_sw128(smem_u32(v_smem), AS_HPLANE, 1024);
    const bool issuer = elect_one();
    bool ok = mbar_wait_all(q_full, 0, wc, DEV_TIMEOUT_ATTN_Q);
    // iteration j issues the scores of tile j and the products of tile j - 1
    for (int j = 0; j <= nkv && ok; ++j) {
      if (j < nkv) {
        const int st = j & 1;
        if (j >= 1 && !mbar_wait_all(s_free, (j - 1) & 1, wc, DEV_TIMEOUT_ATTN_S)) break;
        if (!mbar_wait_all(&k_full[st], (j >> 1) & 1, wc, DEV_TIMEOUT_ATTN_KV)) break;
        tc_fence_after_sync();
        if (issuer) {
          const uint64_t k_desc = k_desc0 + static_cast<uint32_t>(st * (AS_TILE >> 4));
#pragma unroll
          for (int q = 0; q < 6; ++q)
#pragma unroll
            for (int k = 0; k < AS_D / 16; ++k)
              mma_f16_ss(s_tmem, q_desc + PA[q] * PL + 2 * k, k_desc + PB[q] * PL + 2 * k, IDESC_S, (q | k) != 0);
          mma_commit(&k_empty[st]);
          mma_commit(s_full);
        }
      }
      if (j >= 1) {
        const int jj = j - 1;
        if (!mbar_wait_all(p_ready, jj & 1, wc, DEV_TIMEOUT_ATTN_P)) break;
        for (int hf = 0; hf < 2; ++hf) {
          if (!mbar_wait_all(&v_full[hf], jj & 1, wc, DEV_TIMEOUT_ATTN_KV)) { ok = false; break; }
          tc_fence_after_sync();
          if (issuer) {
            const uint64_t v_desc = v_desc0 + static_cast<uint32_t>(hf * (AS_TILE / 2 >> 4));
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // 16 keys: 8 columns of bf16 pairs, 16 rows of V (128 B each)
              const uint64_t vk = v_desc + static_cast<uint64_t>((k * 16 * 128) >> 4);
              const uint32_t pk = p_tmem + 32 * hf + 8 * k;
              mma_f16_ts(o_tmem, pk, vk, IDESC_O3, (hf | k) != 0);
              mma_f16_ts(o_tmem + 64, pk + 64, vk, IDESC_O2, 1);
              mma_f16_ts(o_tmem + 128, pk + 128, vk, IDESC_O1, 1);
            }
            mma_commit(&v_empty[hf]);
          }
        }
        if (ok && issuer) mma_commit(pv_done);
      }
    }
  } else {
    // ------------------------------ softmax + output --------------------------
    const int quad = warp & 3, row = quad * 32 + lane;
    const int half = (warp - 2) >> 2;  // keys 64 * half .. + 63 of a tile, output columns 32 * half .. + 31
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t s_tmem = lane_base + AS_S_COL + 64 * half, p_tmem = lane_base + AS_P_COL + 32 * half,
                   o_tmem = lane_base + AS_O_COL + 32 * half;
    const float c = a.c;
    // The exponentials refer to mc, the running maximum times c as rounded: 2^(s c - mc) has one rounding, and
    // the rounding of mc is the same factor in every term of the row.
    float m = -INFINITY, mc = -INFINITY, l = 0.f;
    float2 o[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] = make_float2(0.f, 0.f);
    // o += the finished products of a tile
    auto add_acc = [&]() {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t a0[16], a1[16], a2[16];
        tmem_ld_32x32b_x16(o_tmem + 16 * g, a0);
        tmem_ld_32x32b_x16(o_tmem + 64 + 16 * g, a1);
        tmem_ld_32x32b_x16(o_tmem + 128 + 16 * g, a2);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          auto pair = [&](const uint32_t (&v)[16]) {
            return make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
          };
          o[8 * g + i] = __fadd2_rn(o[8 * g + i], __fadd2_rn(pair(a0), __fadd2_rn(pair(a1), pair(a2))));
        }
      }
    };
    // this row's value of the other half's thread (slot: alternating buffers, see below)
    auto exchange = [&](int n, float v, float& other) -> bool {
      float* buf = s_max + (n & 1) * 2 * AS_BM;
      buf[half * AS_BM + row] = v;
      __syncwarp();
      if (lane == 0) mbar_arrive(&xchg[quad]);  // release: the warp's writes before it are visible to the waiter
      if (!mbar_wait_warp(&xchg[quad], n & 1, wc, DEV_TIMEOUT_ATTN_S)) return false;
      __syncwarp();
      // a slot is written again two exchanges later, after this warp's next arrival
      other = buf[(half ^ 1) * AS_BM + row];
      return true;
    };
    bool ok = true;
    for (int j = 0; j < nkv; ++j) {
      if (!mbar_wait_warp(s_full, j & 1, wc, DEV_TIMEOUT_ATTN_S)) { ok = false; break; }
      tc_fence_after_sync();
      uint32_t r[2][32];
      tmem_ld_32x32b_x32(s_tmem, r[0]);
      tmem_ld_32x32b_x32(s_tmem + 32, r[1]);
      tmem_wait_ld();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free);
      const int key0 = j * AS_BN + 64 * half;
      if (key0 + 64 > T) {  // keys >= T do not exist
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + 32 * q + i >= T) r[q][i] = 0xff800000u;
      }
      float mx[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t* v = &r[q >> 1][(q & 1) * 16];
        mx[q] = fmaxf(__uint_as_float(v[0]), __uint_as_float(v[1]));
#pragma unroll
        for (int i = 2; i < 16; i += 2) mx[q] = fmax3(mx[q], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      }
      const float own = fmaxf(fmax3(mx[0], mx[1], mx[2]), mx[3]);
      float other;
      if (!exchange(j, own, other)) { ok = false; break; }
      m = fmax3(m, own, other);
      const float mc_new = m * c;
      const float alpha = ex2_f32(mc - mc_new);
      mc = mc_new;
      const float2 c2 = make_float2(c, c), nm2 = make_float2(-mc, -mc);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      uint32_t ph[32], pm[32], pl[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        float2 p = __ffma2_rn(make_float2(__uint_as_float(r[i >> 4][(2 * i) & 31]),
                                          __uint_as_float(r[i >> 4][(2 * i + 1) & 31])), c2, nm2);
        p.x = ex2_f32(p.x);
        p.y = ex2_f32(p.y);
        sum[i & 1] = __fadd2_rn(sum[i & 1], p);
        split3_x2(p.x, p.y, ph[i], pm[i], pl[i]);
      }
      l = fmaf(l, alpha, (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y));
      if (j >= 1) {
        if (!mbar_wait_warp(pv_done, (j - 1) & 1, wc, DEV_TIMEOUT_ATTN_O)) { ok = false; break; }
        tc_fence_after_sync();
        add_acc();
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = __fmul2_rn(o[i], make_float2(alpha, alpha));
      }
      tmem_st_32x32b_x32(p_tmem, ph);
      tmem_st_32x32b_x32(p_tmem + 64, pm);
      tmem_st_32x32b_x32(p_tmem + 128, pl);
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
    }
    float l_other = 0.f;
    if (ok && exchange(nkv, l, l_other) && mbar_wait_warp(pv_done, (nkv - 1) & 1, wc, DEV_TIMEOUT_ATTN_O)) {
      tc_fence_after_sync();
      add_acc();
      const int t = q0 + row;
      const bool ctx = t < a.Tc;
      bf16* out = ctx ? a.out_c : a.out_x;
      if (t < T && out) {
        const int rows = ctx ? a.Tc : T - a.Tc;
        const long plane = static_cast<long>(a.B) * rows * a.E;
        bf16* dst = out + (static_cast<long>(b) * rows + (ctx ? t : t - a.Tc)) * a.E + h * AS_D + 32 * half;
        const float inv = 1.0f / (half ? l_other + l : l + l_other);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 uh, um, ul;
          const float2* v = o + 4 * i;
          split3_x2(v[0].x * inv, v[0].y * inv, uh.x, um.x, ul.x);
          split3_x2(v[1].x * inv, v[1].y * inv, uh.y, um.y, ul.y);
          split3_x2(v[2].x * inv, v[2].y * inv, uh.z, um.z, ul.z);
          split3_x2(v[3].x * inv, v[3].y * inv, uh.w, um.w, ul.w);
          reinterpret_cast<uint4*>(dst)[i] = uh;
          reinterpret_cast<uint4*>(dst + plane)[i] = um;
          reinterpret_cast<uint4*>(dst + 2 * plane)[i] = ul;
        }
      }
    }
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*s_abort) drain_after_abort();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

int launch_attention_split(const AttnProblem* p, int n, int B, int NH, int* dev_status, cudaStream_t stream) {
  if (n < 1 || n > 2 || NH > 65535) {
    set_last_error("attention_split: one or two problems, NH at most 65535");
    return ST_UNSUPPORTED;
  }
  const int E = NH * AS_D;
  static std::mutex attr_mutex;
  static bool attr_done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (!attr_done[dev]) {
      cudaError_t e = cudaFuncSetAttribute(attention_split_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           AS_SMEM_BYTES);
      if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(attention_split)");
      attr_done[dev] = true;
    }
  }
  CUtensorMap tm[2];
  SplitAttnArgs a[2];
  int grid[2] = {0, 0};
  for (int i = 0; i < n; ++i) {
    const AttnProblem& q = p[i];
    if (!q.qkv || !q.out_x || B <= 0 || q.T <= 0 || NH <= 0 || q.Tc < 0 || q.Tc > q.T ||
        (reinterpret_cast<uintptr_t>(q.qkv) & 15) || (reinterpret_cast<uintptr_t>(q.out_x) & 15) ||
        (reinterpret_cast<uintptr_t>(q.out_c) & 15)) {
      set_last_error("attention_split: invalid argument (B %d T %d NH %d Tc %d)", B, q.T, NH, q.Tc);
      return ST_INVALID_ARG;
    }
    int rc = encode_tmap_3d(&tm[i], q.qkv, 2, 3ull * E, (uint64_t)q.T, 3ull * B, 3ull * E * 2,
                            (uint64_t)q.T * 3ull * E * 2, AS_D, 64, 1);
    if (rc) return rc;
    a[i].B = B; a[i].T = q.T; a[i].NH = NH; a[i].Tc = q.Tc; a[i].E = E;
    a[i].out_c = q.out_c;
    a[i].out_x = q.out_x;
    a[i].c = q.scale * 1.4426950408889634f;
    a[i].status = dev_status;
    grid[i] = (q.T + AS_BM - 1) / AS_BM;
  }
  for (int b0 = 0; b0 < B; b0 += 65535) {
    a[0].b0 = a[1].b0 = b0;
    launch_dependent(attention_split_tcgen05_kernel, dim3(grid[0] + grid[1], NH, B - b0 < 65535 ? B - b0 : 65535),
                     AS_THREADS, AS_SMEM_BYTES, stream, tm[0], tm[n - 1], a[0], a[n - 1], grid[0]);
    int rc = after_launch("attention_split_tcgen05_kernel");
    if (rc) return rc;
  }
  return ST_OK;
}

}  // namespace sd3
