// Skinny linear: M = batch rows against a large weight matrix,
//   out[b, n] = act(sum_k in[b, k] W[n, k] + bias[n] + add[b, n]),   W: (N, K) bf16 or fp32.
//
// The weights are read once and there is next to no arithmetic, so the kernel is
// an HBM stream.  A producer warp keeps a ring of shared-memory stages full with
// bulk copies (one per weight row and K chunk, 1536 bytes), eight consumer warps
// own R rows each and form the dot products of up to eight samples from shared
// memory (a weight is read once per warp, an activation once per R rows).  Bytes in
// flight then do not depend on registers or on how long the arithmetic of a slab
// takes, as they did in the kernel this replaced (weights straight into registers, loads
// and arithmetic in turn).  Measured, before -> after, 1 / 8 samples: 502272 x 1536 fp32
// 721 / 1389 -> 595 / 1285 us (5.2 / 2.4 TB/s of weights), 23040 x 1536 (one dual block) fp32 48 / 85 ->
// 34 / 68 us, bf16 43 / 72 -> 22 / 57 us.  With eight samples the activations' shared-memory reads bound it.
//
// The order of a sum is part of the result: it decides the last bits of the conditioning vector, some of
// which then round to the neighbouring bf16 and reach every block.  With bf16 weights lane l adds the
// products of k = 256 i + 8 l + j in the order of i and j (16 bytes of a weight row per lane and step), then
// the lanes are added pairwise, 16 apart first: the bits of the kernel that this one replaced.  With fp32 weights a lane
// takes 4 consecutive elements, k = 128 i + 4 l + j, also 16 bytes; 8 would cost 595 -> 937 us on
// 502272 x 1536 (two loads per row and step, shorter chunks), and the fp32 model's GEMMs
// sum in another order than before in any case.
//
// R = 4 for matrices that give every SM work for several rounds, R = 1 for the
// small ones (1536 rows: 192 CTAs instead of 48, the chain of K chunks is what they take).
//
// In a chain of launches whose weights no kernel writes (w_static), the first ring of weights is
// requested before the wait for the preceding kernel, which hides the HBM latency of the small layers.
#include <mutex>

#include "kernels.h"
#include "ptx.cuh"

namespace sd3 {

int device_sm_count();

namespace {

constexpr int SK_WARPS = 8;                    // consumer warps
constexpr int SK_THREADS = 32 * (SK_WARPS + 1);
constexpr int SK_CHUNK = 1536;                 // bytes of a weight row per stage

template <typename WT, int R, int BC>
struct SkinnyCfg {
  static constexpr int KC = SK_CHUNK / static_cast<int>(sizeof(WT));  // K elements per stage
  static constexpr int VK = 16 / static_cast<int>(sizeof(WT));        // consecutive elements of K per lane and step
  static constexpr int ROWS = SK_WARPS * R;
  static constexpr int W_BYTES = ROWS * SK_CHUNK;
  static constexpr int X_BYTES = BC * KC * 4;
  static constexpr int STAGE = W_BYTES + X_BYTES;
  static constexpr int STAGES = R == 1 ? 6 : 3;  // at most 3 * 72 KiB or 6 * 36 KiB
  static constexpr int SMEM = STAGES * STAGE + 128;
};

struct SkinnyArgs {
  const float* in;
  long ld_in;
  const void* W;
  const float* bias;
  const float* add;
  long ld_add;
  float* out;
  long ld_out;
  int B, N, K, act_out, w_static;
  int* status;
};

__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem_dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// elements 2 i and 2 i + 1 of the words of a packed weight vector as floats
__device__ __forceinline__ float4 unpack4(uint32_t a, uint32_t b) {
  return make_float4(__uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u), __uint_as_float(b << 16),
                     __uint_as_float(b & 0xffff0000u));
}
__device__ __forceinline__ float dot4(const float4& x, const float4& w, float acc) {
  return fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, acc))));
}

template <typename WT, int R, int BC>
__global__ void __launch_bounds__(SK_THREADS, 1) skinny_stream_kernel(const SkinnyArgs a) {
  using Cfg = SkinnyCfg<WT, R, BC>;
  constexpr int KC = Cfg::KC, VK = Cfg::VK, STAGES = Cfg::STAGES;
  extern __shared__ __align__(128) uint8_t sk_smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(sk_smem + STAGES * Cfg::STAGE);
  uint64_t* empty = full + STAGES;
  int* s_abort = reinterpret_cast<int*>(empty + STAGES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], SK_WARPS);
    }
    *s_abort = 0;
    fence_barrier_init();
  }
  __syncthreads();
  const WaitCtx wc{s_abort, a.status};
  const int kchunks = (a.K + KC - 1) / KC;
  const int groups = (a.N + Cfg::ROWS - 1) / Cfg::ROWS;
  const int mine = (groups - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int per_pass = mine * kchunks;                 // stages of one pass over the weights
  const int total = per_pass * ((a.B + BC - 1) / BC);  // one pass per BC samples

  if (warp == SK_WARPS) {
    // ------------------------------ producer warp -----------------------------
    const WT* W = static_cast<const WT*>(a.W);
    auto issue_w = [&](int it) {  // expects the whole stage's bytes, copies the weight rows
      const int s = it % STAGES, r = it % per_pass;
      const int n0 = (static_cast<int>(blockIdx.x) + (r / kchunks) * static_cast<int>(gridDim.x)) * Cfg::ROWS;
      const int k0 = (r % kchunks) * KC, len = min(KC, a.K - k0);
      const int rows = min(Cfg::ROWS, a.N - n0), nb = min(BC, a.B - (it / per_pass) * BC);
      if (lane == 0) mbar_expect_tx(&full[s], rows * len * static_cast<int>(sizeof(WT)) + nb * len * 4);
      __syncwarp();
      for (int i = lane; i < rows; i += 32)
        bulk_load(sk_smem + s * Cfg::STAGE + i * SK_CHUNK, W + static_cast<long>(n0 + i) * a.K + k0,
                  len * static_cast<int>(sizeof(WT)), &full[s]);
    };
    auto issue_x = [&](int it) {
      const int s = it % STAGES, r = it % per_pass, b0 = (it / per_pass) * BC;
      const int k0 = (r % kchunks) * KC, len = min(KC, a.K - k0), nb = min(BC, a.B - b0);
      if (lane < nb)
        bulk_load(sk_smem + s * Cfg::STAGE + Cfg::W_BYTES + lane * KC * 4, a.in + (b0 + lane) * a.ld_in + k0, len * 4,
                  &full[s]);
    };
    const int first = min(total, STAGES);
    if (!a.w_static) grid_dep_wait();
    for (int it = 0; it < first; ++it) issue_w(it);
    if (a.w_static) grid_dep_wait();
    grid_dep_launch();
    for (int it = 0; it < first; ++it) issue_x(it);
    for (int it = first; it < total; ++it) {
      if (!mbar_wait_warp(&empty[it % STAGES], ((it / STAGES) - 1) & 1, wc, DEV_TIMEOUT_EMPTY)) break;
      issue_w(it);
      issue_x(it);
    }
  } else {
    // ------------------------------ consumer warps ----------------------------
    grid_dep_wait();
    int it = 0;
    bool ok = true;
    for (int b0 = 0; b0 < a.B && ok; b0 += BC) {
      for (int g = 0; g < mine && ok; ++g) {
        float acc[R][BC];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int b = 0; b < BC; ++b) acc[r][b] = 0.f;
        for (int kc = 0; kc < kchunks; ++kc, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait_warp(&full[s], (it / STAGES) & 1, wc, DEV_TIMEOUT_FULL)) { ok = false; break; }
          const int len = min(KC, a.K - kc * KC);
          const uint8_t* st = sk_smem + s * Cfg::STAGE;
          const float* xs = reinterpret_cast<const float*>(st + Cfg::W_BYTES);
#pragma unroll
          for (int i = 0; i < KC / (32 * VK); ++i) {
            const int k = 32 * VK * i + VK * lane;
            if (k < len) {  // K is a multiple of 8
              uint4 w[R];
#pragma unroll
              for (int r = 0; r < R; ++r)
                w[r] = *reinterpret_cast<const uint4*>(reinterpret_cast<const WT*>(st + (warp * R + r) * SK_CHUNK) + k);
#pragma unroll
              for (int b = 0; b < BC; ++b) {
                const float* xp = xs + b * KC + k;
                if constexpr (VK == 4) {
                  const float4 x = load4(xp);
#pragma unroll
                  for (int r = 0; r < R; ++r)
                    acc[r][b] = dot4(x, make_float4(__uint_as_float(w[r].x), __uint_as_float(w[r].y),
                                                    __uint_as_float(w[r].z), __uint_as_float(w[r].w)), acc[r][b]);
                } else {
                  // 32 bytes per lane: every other group of four lanes reads its halves in the opposite
                  // order, so that eight lanes cover all banks
                  const int swap = lane & 4;
                  const float4 u = load4(xp + swap), v = load4(xp + 4 - swap);
                  const float4 x0 = swap ? v : u, x1 = swap ? u : v;
#pragma unroll
                  for (int r = 0; r < R; ++r)
                    acc[r][b] = dot4(x1, unpack4(w[r].z, w[r].w), dot4(x0, unpack4(w[r].x, w[r].y), acc[r][b]));
                }
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[s]);
        }
        if (!ok) break;
        const long n0 = (static_cast<long>(blockIdx.x) + static_cast<long>(g) * gridDim.x) * Cfg::ROWS + warp * R;
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
          for (int b = 0; b < BC; ++b) {
            const float v = warp_sum(acc[r][b]);
            if (lane == (r * BC + b) % 32 && n0 + r < a.N && b0 + b < a.B) {
              float o = v + (a.bias ? a.bias[n0 + r] : 0.f);
              if (a.add) o += a.add[(b0 + b) * a.ld_add + n0 + r];
              if (a.act_out == 1) o = o / (1.f + expf(-o));
              a.out[(b0 + b) * a.ld_out + n0 + r] = o;
            }
          }
        }
      }
    }
  }
  __syncthreads();
  if (*s_abort) drain_after_abort();
}

template <typename WT, int R, int BC>
int launch_skinny_inst(const SkinnyArgs& a, cudaStream_t stream) {
  using Cfg = SkinnyCfg<WT, R, BC>;
  auto kern = skinny_stream_kernel<WT, R, BC>;
  static std::mutex attr_mutex;
  static bool attr_done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (!attr_done[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
      if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(skinny_linear)");
      attr_done[dev] = true;
    }
  }
  const int groups = (a.N + Cfg::ROWS - 1) / Cfg::ROWS;
  const int most = device_sm_count();
  launch_dependent(kern, groups < most ? groups : most, SK_THREADS, Cfg::SMEM, stream, a);
  return after_launch("skinny_stream_kernel");
}

template <typename WT, int R>
int launch_skinny_batch(const SkinnyArgs& a, cudaStream_t stream) {
  if (a.B == 1) return launch_skinny_inst<WT, R, 1>(a, stream);
  if (a.B == 2) return launch_skinny_inst<WT, R, 2>(a, stream);
  if (a.B <= 4) return launch_skinny_inst<WT, R, 4>(a, stream);
  return launch_skinny_inst<WT, R, 8>(a, stream);
}

}  // namespace

int launch_skinny_linear(const float* in, long ld_in, const void* W, int w_f32, const float* bias, const float* add,
                         long ld_add, float* out, long ld_out, int B, int N, int K, int act_out, int* dev_status,
                         cudaStream_t stream, bool w_static) {
  if (!in || !W || !out || B <= 0 || N <= 0 || K <= 0 || (K & 7) || (ld_in & 3) ||
      (reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(W) & 15)) {
    set_last_error("skinny_linear: invalid argument (K %d must be a multiple of 8, operands 16-byte aligned)", K);
    return ST_INVALID_ARG;
  }
  const SkinnyArgs a = {in, ld_in, W, bias, add, ld_add, out, ld_out, B, N, K, act_out, w_static ? 1 : 0,
                        dev_status};
  // R = 4 once 32-row groups give every SM at least two
  const bool large = N >= 64L * device_sm_count();
  if (w_f32) return large ? launch_skinny_batch<float, 4>(a, stream) : launch_skinny_batch<float, 1>(a, stream);
  return large ? launch_skinny_batch<bf16, 4>(a, stream) : launch_skinny_batch<bf16, 1>(a, stream);
}

}  // namespace sd3
