// HBM-bound kernels of the denoiser forward: LayerNorm + AdaLN modulation,
// timestep / position embeddings, patch gathering,
// casts and transposes for weight packing, and a stand-alone per-head RMSNorm.
// All of them are coalesced, 128-bit vectorised and warp-shuffle reduced.
//
// Reference counterparts: layernorm_forward_kernel6 (cuda/dit.cu:17-75) and
// scale_and_shift3 (cuda/dit.cu:357-374) -> ln_modulate_kernel (one pass, both
// modulations of a dual block at once); partial_linear_cuda launched 15x per
// block with M = batch (cuda/dit.cu:102-354) -> skinny.cu and, in bf16 models, one
// GEMM for every block's AdaLN vectors (engine.cu); sinusoidal_embedding
// (modules.cpp:920-944); positional_embedding2D + crop
// (modules.cpp:946-995); conv2d im2col side of PatchEmbedding
// (modules.cpp:1037-1117); rmsnorm_key_query_kernel2 (cuda/dit.cu:384-447).
#include "kernels.h"
#include "launch_rules.h"
#include "ptx.cuh"
#include "split3.cuh"

namespace sd3 {

int device_sm_count();

namespace {

// ----------------------------------------------------------------------------
// LayerNorm + modulate.  One warp per row, the row lives in registers (fewer rows: one CTA per row, further down).
// ----------------------------------------------------------------------------
// OUT: 0 bf16, 1 fp32, 2 e4m3 (operand of an FP8 GEMM, converted as is), 3 three bf16 planes of
// rows * E elements (operand of a split fp32 GEMM)
//
// A CTA of 8 warps owns 8 * rpw consecutive rows (rpw per warp, at most 8; fewer
// for small inputs so that the grid still covers the GPU).  The
// modulation vectors (1 + scale, shift; two pairs for DUAL) of the sample its
// first row belongs to are staged in shared memory once: re-reading them from
// global memory for every row (12 KB per 6 KB row, all L1 hits) cost a quarter
// of the kernel's bandwidth.  Rows of another sample (a CTA that straddles a
// sample boundary) read theirs from global memory.
//
// One launch takes one or two problems (the image and the context rows of a block,
// whose LayerNorms stand next to each other everywhere): at small sizes the kernel
// is one chain of latencies (launch, row, two reductions, store; 7 us for 256 rows),
// and two of them in a row cost twice that.  The first row is requested before the
// barrier behind the staging.  Measured (whole forward, one image): 256x256 3510 -> 3326 us,
// 1024x1024 14.18 -> 13.96 ms.  Three CTAs per SM for the plane output, whose splits need the registers.
constexpr int LN_MAX_ROWS_PER_WARP = 8;
constexpr int LN_WARPS = 8;

// four consecutive values as three bf16 planes
__device__ __forceinline__ void store4_split(bf16* p, long plane, const float4& o) {
  uint2 h, m, l;
  split3_x2(o.x, o.y, h.x, m.x, l.x);
  split3_x2(o.z, o.w, h.y, m.y, l.y);
  *reinterpret_cast<uint2*>(p) = h;
  *reinterpret_cast<uint2*>(p + plane) = m;
  *reinterpret_cast<uint2*>(p + 2 * plane) = l;
}

template <int OUT>
__device__ __forceinline__ void ln_store4(void* out, long row, long rows, int E, int i, const float4& o) {
  if constexpr (OUT == 3) {
    store4_split(static_cast<bf16*>(out) + row * E + 4 * i, rows * E, o);
  } else if constexpr (OUT == 1) {
    reinterpret_cast<float4*>(static_cast<float*>(out) + row * E)[i] = o;
  } else if constexpr (OUT == 2) {
    reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(out) + row * E)[i] = pack_e4m3x4(o.x, o.y, o.z, o.w);
  } else {
    uint2 u;
    u.x = pack_bf16x2(o.x, o.y);
    u.y = pack_bf16x2(o.z, o.w);
    reinterpret_cast<uint2*>(static_cast<bf16*>(out) + row * E)[i] = u;
  }
}

template <int MAXV, int OUT, bool DUAL>
__global__ void __launch_bounds__(LN_WARPS * 32, OUT == 3 ? 3 : 4)
ln_modulate_kernel(const __grid_constant__ LnProblem pa, const __grid_constant__ LnProblem pb, const unsigned grid_a, int E, float eps, long mod_stride,
                   int rpw) {
  extern __shared__ float4 ln_smem[];  // [1 + scale1 | shift1 | 1 + scale2 | shift2], E floats each
  grid_dep_wait();
  grid_dep_launch();
  const bool second = blockIdx.x >= grid_a;
  const LnProblem& p = second ? pb : pa;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = E >> 2;
  const int T = p.T;
  const long rows = static_cast<long>(p.B) * T;
  const bool dual = DUAL && p.out2 != nullptr;
  const long row0 = static_cast<long>(second ? blockIdx.x - grid_a : blockIdx.x) * (LN_WARPS * rpw);
  const int b_cta = static_cast<int>(row0 / T);
  float4* s_sc1 = ln_smem;
  float4* s_sh1 = ln_smem + nvec;
  float4* s_sc2 = ln_smem + 2 * nvec;
  float4* s_sh2 = ln_smem + 3 * nvec;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    float4 s = *(reinterpret_cast<const float4*>(p.scale1 + b_cta * mod_stride) + i);
    s.x += 1.f; s.y += 1.f; s.z += 1.f; s.w += 1.f;
    s_sc1[i] = s;
    s_sh1[i] = *(reinterpret_cast<const float4*>(p.shift1 + b_cta * mod_stride) + i);
    if (dual) {
      float4 s2 = *(reinterpret_cast<const float4*>(p.scale2 + b_cta * mod_stride) + i);
      s2.x += 1.f; s2.y += 1.f; s2.z += 1.f; s2.w += 1.f;
      s_sc2[i] = s2;
      s_sh2[i] = *(reinterpret_cast<const float4*>(p.shift2 + b_cta * mod_stride) + i);
    }
  }
#pragma unroll 1
  for (int rw = 0; rw < rpw; ++rw) {
    const long row = row0 + static_cast<long>(rw) * LN_WARPS + warp;  // warps interleave rows
    const bool live = row < rows;
    const float4* xr = reinterpret_cast<const float4*>(p.x + row * E);
    float4 v[MAXV];
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = lane + 32 * j;
      if (live && i < nvec) {
        v[j] = xr[i];
        sum += (v[j].x + v[j].y) + (v[j].z + v[j].w);
      } else {
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (rw == 0) __syncthreads();  // the staged vectors are complete; the first row was requested before
    if (!live) break;
    const float mean = warp_sum(sum) / static_cast<float>(E);
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec) {
        const float a = v[j].x - mean, bq = v[j].y - mean, c = v[j].z - mean, d = v[j].w - mean;
        sq += (a * a + bq * bq) + (c * c + d * d);
      }
    }
    const int b = static_cast<int>(row / T);
    const float rstd = rsqrtf(warp_sum(sq) / static_cast<float>(E) + eps);
    const bool cached = b == b_cta;  // warp-uniform
    const long moff = static_cast<long>(b) * mod_stride;  // used by rows of another sample only
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec) {
        float4 n;
        n.x = (v[j].x - mean) * rstd;
        n.y = (v[j].y - mean) * rstd;
        n.z = (v[j].z - mean) * rstd;
        n.w = (v[j].w - mean) * rstd;
        {
          float4 s, h;
          if (cached) {
            s = s_sc1[i]; h = s_sh1[i];
          } else {
            s = *(reinterpret_cast<const float4*>(p.scale1 + moff) + i);
            h = *(reinterpret_cast<const float4*>(p.shift1 + moff) + i);
            s.x += 1.f; s.y += 1.f; s.z += 1.f; s.w += 1.f;
          }
          float4 o;
          o.x = fmaf(n.x, s.x, h.x);
          o.y = fmaf(n.y, s.y, h.y);
          o.z = fmaf(n.z, s.z, h.z);
          o.w = fmaf(n.w, s.w, h.w);
          ln_store4<OUT>(p.out1, row, rows, E, i, o);
        }
        if (dual) {
          float4 s, h;
          if (cached) {
            s = s_sc2[i]; h = s_sh2[i];
          } else {
            s = *(reinterpret_cast<const float4*>(p.scale2 + moff) + i);
            h = *(reinterpret_cast<const float4*>(p.shift2 + moff) + i);
            s.x += 1.f; s.y += 1.f; s.z += 1.f; s.w += 1.f;
          }
          float4 o;
          o.x = fmaf(n.x, s.x, h.x);
          o.y = fmaf(n.y, s.y, h.y);
          o.z = fmaf(n.z, s.z, h.z);
          o.w = fmaf(n.w, s.w, h.w);
          ln_store4<OUT>(p.out2, row, rows, E, i, o);
        }
      }
    }
  }
}

// The same with a CTA of four warps per row: the row and its modulation vectors are requested at once and one memory latency
// is exposed, where the kernel above stages the vectors first.  MULTI: the CTA takes per_cta consecutive rows, keeps
// the vectors in registers (read for every row, two modulations' are four times the row's bytes, all from L2) and
// has the next row under way while it forms one.  The sums are formed in the order of the kernel above (each lane adds its
// quads in order, then the lanes' tree): the same bits.  Bound by latency at a thousand rows, by L2 and HBM
// above (5.9 TB/s at 35432 rows).  Which sizes take it: ln_kernel (launch_rules.h), with the figures.
template <int OUT, bool DUAL, bool MULTI>
__global__ void __launch_bounds__(128)
ln_modulate_row_kernel(const __grid_constant__ LnProblem pa, const __grid_constant__ LnProblem pb, const unsigned grid_a,
                       int E, float eps, long mod_stride, int per_cta) {
  __shared__ float part[2][LN_ROW_QUADS][32];
  grid_dep_wait();
  grid_dep_launch();
  const bool second = blockIdx.x >= grid_a;
  const LnProblem& p = second ? pb : pa;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = E >> 2;
  const long rows = static_cast<long>(p.B) * p.T;
  const long row0 = static_cast<long>(second ? blockIdx.x - grid_a : blockIdx.x) * (MULTI ? per_cta : 1);
  const long row_end = !MULTI ? row0 + 1 : row0 + per_cta < rows ? row0 + per_cta : rows;
  const bool dual = DUAL && p.out2 != nullptr;
  constexpr int NV = LN_ROW_QUADS / 4;  // quads of a thread: j = NV * warp + t, elements 4 (lane + 32 j)
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 v[NV], next[MULTI ? NV : 1], sc1[NV], sh1[NV], sc2[DUAL ? NV : 1], sh2[DUAL ? NV : 1];
  long b_now = row0 / p.T, b_end = (b_now + 1) * p.T;  // the sample of the current row, its first row past the end
  auto load = [&](float4* x, long row, bool mod) {
    const long moff = b_now * mod_stride;
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      const int i = lane + 32 * (NV * warp + t);
      const bool in = i < nvec;
      if (x != nullptr) x[t] = in ? *(reinterpret_cast<const float4*>(p.x + row * E) + i) : z4;
      if (!mod) continue;
      sc1[t] = in ? *(reinterpret_cast<const float4*>(p.scale1 + moff) + i) : z4;
      sh1[t] = in ? *(reinterpret_cast<const float4*>(p.shift1 + moff) + i) : z4;
      if constexpr (DUAL) {
        sc2[t] = in && dual ? *(reinterpret_cast<const float4*>(p.scale2 + moff) + i) : z4;
        sh2[t] = in && dual ? *(reinterpret_cast<const float4*>(p.shift2 + moff) + i) : z4;
      }
    }
  };
  load(v, row0, true);
  auto row_sum = [&](float (&buf)[LN_ROW_QUADS][32]) {
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < LN_ROW_QUADS; ++j) s += buf[j][lane];
    return warp_sum(s);
  };
#pragma unroll 1
  for (long row = row0; row < row_end; ++row) {
    if constexpr (MULTI) {
      if (row + 1 < row_end) load(next, row + 1, false);  // under way while this row is formed
      if (row == b_end) {
        b_end += p.T;
        ++b_now;
        load(nullptr, 0, true);
      }
    }
#pragma unroll
    for (int t = 0; t < NV; ++t) part[0][NV * warp + t][lane] = (v[t].x + v[t].y) + (v[t].z + v[t].w);
    const float mean = row_sum(part[0]) / static_cast<float>(E);
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      const float a = v[t].x - mean, b = v[t].y - mean, c = v[t].z - mean, d = v[t].w - mean;
      part[1][NV * warp + t][lane] = lane + 32 * (NV * warp + t) < nvec ? (a * a + b * b) + (c * c + d * d) : 0.f;
    }
    const float rstd = rsqrtf(row_sum(part[1]) / static_cast<float>(E) + eps);
    auto modulate = [&](const float4& x, const float4& s, const float4& h) {
      return make_float4(fmaf((x.x - mean) * rstd, s.x + 1.f, h.x), fmaf((x.y - mean) * rstd, s.y + 1.f, h.y),
                         fmaf((x.z - mean) * rstd, s.z + 1.f, h.z), fmaf((x.w - mean) * rstd, s.w + 1.f, h.w));
    };
#pragma unroll
    for (int t = 0; t < NV; ++t) {
      const int i = lane + 32 * (NV * warp + t);
      if (i < nvec) {
        ln_store4<OUT>(p.out1, row, rows, E, i, modulate(v[t], sc1[t], sh1[t]));
        if constexpr (DUAL) {
          if (dual) ln_store4<OUT>(p.out2, row, rows, E, i, modulate(v[t], sc2[t], sh2[t]));
        }
      }
      if constexpr (MULTI) v[t] = next[t];
    }
  }
}

template <int MAXV>
int launch_ln_inst(const LnProblem& a, const LnProblem* b, int E, float eps, long mod_stride, int out_f32,
                   cudaStream_t stream) {
  const long rows_a = static_cast<long>(a.B) * a.T, rows_b = b ? static_cast<long>(b->B) * b->T : 0;
  // rows per warp: as many as keeps at least two CTAs per SM busy
  int rpw = LN_MAX_ROWS_PER_WARP;
  auto ctas = [&](long rows) { return (rows + LN_WARPS * rpw - 1) / (LN_WARPS * rpw); };
  while (rpw > 1 && ctas(rows_a) + ctas(rows_b) < 2L * device_sm_count()) rpw >>= 1;
  const unsigned grid_a = static_cast<unsigned>(ctas(rows_a)), grid = grid_a + static_cast<unsigned>(ctas(rows_b));
  const bool dual = a.out2 != nullptr || (b && b->out2 != nullptr);
  const size_t smem = static_cast<size_t>(E) * 4 * (dual ? 4 : 2);
  const LnProblem pb = b ? *b : a;
  const LnKernel kind = ln_kernel(E, rows_a + rows_b, dual, device_sm_count());
  if (kind != LN_WARP_PER_ROW) {
    const bool multi = kind == LN_ROWS_PER_CTA;
    // rows of a CTA: as many as lets all CTAs be resident at once, up to a limit
    const long resident = 5L * device_sm_count(), most = dual ? 64 : 8;
    const long want = (rows_a + rows_b + resident - 1) / resident;
    const int per = !multi ? 1 : static_cast<int>(want > most ? most : want);
    const unsigned ga = static_cast<unsigned>((rows_a + per - 1) / per);
    const dim3 row_ctas(ga + static_cast<unsigned>((rows_b + per - 1) / per));
#define SD3_LN_ROW_INST(F32, DUALV, MULTIV)                                                                              \
  launch_dependent(ln_modulate_row_kernel<F32, DUALV, MULTIV>, row_ctas, 128, 0, stream, a, pb, ga, E, eps, mod_stride, per)
#define SD3_LN_ROW(F32)                                     \
  case F32:                                                 \
    if (dual) SD3_LN_ROW_INST(F32, true, true);             \
    else if (multi) SD3_LN_ROW_INST(F32, false, true);      \
    else SD3_LN_ROW_INST(F32, false, false);                \
    break
    switch (out_f32) {
      SD3_LN_ROW(1);
      SD3_LN_ROW(2);
      SD3_LN_ROW(3);
      default:
      SD3_LN_ROW(0);
    }
#undef SD3_LN_ROW
#undef SD3_LN_ROW_INST
    return after_launch("ln_modulate_row_kernel");
  }
#define SD3_LN_LAUNCH(F32)                                                                                               \
  do {                                                                                                                   \
    if constexpr (MAXV != LN_ROW_QUADS) {                                                                                \
      if (dual) {                                                                                                        \
        launch_dependent(ln_modulate_kernel<MAXV, F32, true>, grid, LN_WARPS * 32, smem, stream, a, pb, grid_a, E,       \
                         eps, mod_stride, rpw);                                                                          \
        break;                                                                                                           \
      }                                                                                                                  \
    }                                                                                                                    \
    launch_dependent(ln_modulate_kernel<MAXV, F32, false>, grid, LN_WARPS * 32, smem, stream, a, pb, grid_a, E, eps,     \
                     mod_stride, rpw);                                                                                   \
  } while (0)
  switch (out_f32) {
    case 1: SD3_LN_LAUNCH(1); break;
    case 2: SD3_LN_LAUNCH(2); break;
    case 3: SD3_LN_LAUNCH(3); break;
    default: SD3_LN_LAUNCH(0);
  }
#undef SD3_LN_LAUNCH
  return after_launch("ln_modulate_kernel");
}

__global__ void sinusoidal_kernel(const float* t, float* out, int B,
                                  int dim) {
  grid_dep_wait();
  grid_dep_launch();
  const int half = dim / 2;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= B * half) return;
  const int b = idx / half, i = idx % half;
  // same fp32 operation order as the reference: exp(-ln(1e4) * i / half), then t * f
  const float f = expf(-9.2103403719761836f * static_cast<float>(i) / static_cast<float>(half));
  const float a = t[b] * f;
  out[static_cast<long>(b) * dim + i] = cosf(a);
  out[static_cast<long>(b) * dim + half + i] = sinf(a);
}

__global__ void pos_table_kernel(float* __restrict__ table, int h, int w, int E, int pmax,
                                 int base_size) {
  const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int q = E / 4;
  const long total = static_cast<long>(h) * w * q;
  if (idx >= total) return;
  const int i = static_cast<int>(idx % q);
  const long tok = idx / q;
  const int s = static_cast<int>(tok % w), r = static_cast<int>(tok / w);
  const int R = r + (pmax - h) / 2, S = s + (pmax - w) / 2;
  const double denom = static_cast<double>(pmax) / static_cast<double>(base_size);
  const double div = 1.0 / pow(10000.0, static_cast<double>(i) / (static_cast<double>(E) / 4.0));
  const double ps = (static_cast<double>(S) / denom) * div;
  const double pr = (static_cast<double>(R) / denom) * div;
  float* o = table + tok * E;
  o[i] = static_cast<float>(sin(ps));
  o[q + i] = static_cast<float>(cos(ps));
  o[2 * q + i] = static_cast<float>(sin(pr));
  o[3 * q + i] = static_cast<float>(cos(pr));
}

template <typename IT, typename OT>
__device__ __forceinline__ OT convert_elem(IT v);
template <> __device__ __forceinline__ float convert_elem<float, float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 convert_elem<float, bf16>(float v) { return __float2bfloat16(v); }
template <> __device__ __forceinline__ float convert_elem<bf16, float>(bf16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ bf16 convert_elem<bf16, bf16>(bf16 v) { return v; }

template <typename IT, bool SPLIT>
__global__ void patchify_kernel(const IT* latent, bf16* out, int B, int C,
                                int H, int W, int p) {
  grid_dep_wait();
  grid_dep_launch();
  const int hp = H / p, wp = W / p;
  const int Kp = C * p * p;
  const long total = static_cast<long>(B) * hp * wp * Kp;
  const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int k = static_cast<int>(idx % Kp);
  const long tok = idx / Kp;
  const int s = static_cast<int>(tok % wp);
  const int r = static_cast<int>((tok / wp) % hp);
  const int b = static_cast<int>(tok / (static_cast<long>(wp) * hp));
  const int pw = k % p, ph = (k / p) % p, c = k / (p * p);
  const long src = ((static_cast<long>(b) * C + c) * H + (r * p + ph)) * W + (s * p + pw);
  if constexpr (SPLIT) {
    uint32_t h, m, l;
    split3_x2(convert_elem<IT, float>(latent[src]), 0.f, h, m, l);
    unsigned short* o = reinterpret_cast<unsigned short*>(out) + idx;
    o[0] = static_cast<unsigned short>(h);
    o[total] = static_cast<unsigned short>(m);
    o[2 * total] = static_cast<unsigned short>(l);
  } else {
    out[idx] = convert_elem<IT, bf16>(latent[src]);
  }
}

template <typename IT, typename OT>
__global__ void cast_kernel(const IT* in, OT* out, long n) {
  grid_dep_wait();
  grid_dep_launch();
  long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x;
  for (; i < n; i += stride) out[i] = convert_elem<IT, OT>(in[i]);
}

template <typename IT, typename OT>
__global__ void transpose_kernel(const IT* __restrict__ in, OT* __restrict__ out, int R, int C) {
  __shared__ float tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int r = r0 + j, c = c0 + threadIdx.x;
    tile[j][threadIdx.x] =
        (r < R && c < C) ? convert_elem<IT, float>(in[static_cast<long>(r) * C + c]) : 0.f;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int c = c0 + j, r = r0 + threadIdx.x;
    if (r < R && c < C)
      out[static_cast<long>(c) * R + r] = convert_elem<float, OT>(tile[threadIdx.x][j]);
  }
}

// VEC: in is aligned to four elements (a caller's captions need not be)
template <typename IT, bool VEC>
__global__ void split3_kernel(const IT* in, bf16* out, long n) {
  grid_dep_wait();
  grid_dep_launch();
  long i = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x * 4;
  for (; i < n; i += stride) {
    float4 f;
    if constexpr (!VEC) {
      f = make_float4(convert_elem<IT, float>(in[i]), convert_elem<IT, float>(in[i + 1]),
                      convert_elem<IT, float>(in[i + 2]), convert_elem<IT, float>(in[i + 3]));
    } else if constexpr (sizeof(IT) == 4) {
      f = *reinterpret_cast<const float4*>(in + i);
    } else {
      const uint2 u = *reinterpret_cast<const uint2*>(in + i);
      f = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                      __uint_as_float(u.y & 0xffff0000u));
    }
    store4_split(out + i, n, f);
  }
}

// 64 rows x 32 columns per CTA: reads rows of 128 bytes, writes rows of 64 bf16 per plane
template <typename IT>
__global__ void transpose_split3_kernel(const IT* __restrict__ in, bf16* __restrict__ out, int R, int C) {
  __shared__ float tile[64][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 64;
  const long plane = static_cast<long>(R) * C;
  for (int j = threadIdx.y; j < 64; j += blockDim.y) {
    const int r = r0 + j, c = c0 + threadIdx.x;
    tile[j][threadIdx.x] = (r < R && c < C) ? convert_elem<IT, float>(in[static_cast<long>(r) * C + c]) : 0.f;
  }
  __syncthreads();
  const int r = r0 + 2 * threadIdx.x;  // R is even
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int c = c0 + j;
    if (r < R && c < C) {
      uint32_t h, m, l;
      split3_x2(tile[2 * threadIdx.x][j], tile[2 * threadIdx.x + 1][j], h, m, l);
      bf16* o = out + static_cast<long>(c) * R + r;
      *reinterpret_cast<uint32_t*>(o) = h;
      *reinterpret_cast<uint32_t*>(o + plane) = m;
      *reinterpret_cast<uint32_t*>(o + 2 * plane) = l;
    }
  }
}

template <typename XT>
__global__ void rmsnorm_heads_kernel(XT* x, long ld, long rows, int col0, int nheads,
                                     int D, const float* w, float eps) {
  grid_dep_wait();
  grid_dep_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long unit = static_cast<long>(blockIdx.x) * (blockDim.x >> 5) + warp;
  if (unit >= rows * nheads) return;
  const long row = unit / nheads;
  const int h = static_cast<int>(unit % nheads);
  XT* p = x + row * ld + col0 + h * D;
  float ss = 0.f;
  for (int i = lane; i < D; i += 32) {
    const float v = convert_elem<XT, float>(p[i]);
    ss += v * v;
  }
  const float r = rsqrtf(warp_sum(ss) / static_cast<float>(D) + eps);
  for (int i = lane; i < D; i += 32) {
    const float v = convert_elem<XT, float>(p[i]) * r * (w ? w[i] : 1.f);
    p[i] = convert_elem<float, XT>(v);
  }
}

}  // namespace

int launch_ln_modulate(const LnProblem& a, const LnProblem* b, int E, float eps, long mod_stride, int out_f32,
                       cudaStream_t stream) {
  for (const LnProblem* p : {&a, b}) {
    if (!p) continue;
    if (!p->x || !p->out1 || !p->shift1 || !p->scale1 || p->B <= 0 || p->T <= 0 || E <= 0 || (E & 3) ||
        (mod_stride & 3)) {
      set_last_error("ln_modulate: invalid argument (E %d must be a multiple of 4)", E);
      return ST_INVALID_ARG;
    }
    if (p->out2 && (!p->shift2 || !p->scale2)) {
      set_last_error("ln_modulate: second output needs its own shift/scale");
      return ST_INVALID_ARG;
    }
  }
  const int nvec = E / 4;
#define SD3_LN_CASE(MV) \
  if (nvec <= 32 * MV) return launch_ln_inst<MV>(a, b, E, eps, mod_stride, out_f32, stream)
  SD3_LN_CASE(2);
  SD3_LN_CASE(6);
  SD3_LN_CASE(12);
  SD3_LN_CASE(16);
  SD3_LN_CASE(32);
#undef SD3_LN_CASE
  set_last_error("ln_modulate: E %d too large (max 4096)", E);
  return ST_UNSUPPORTED;
}

int launch_sinusoidal(const float* t, float* out, int B, int dim, cudaStream_t stream) {
  if (!t || !out || B <= 0 || dim <= 0 || (dim & 1)) {
    set_last_error("sinusoidal: invalid argument");
    return ST_INVALID_ARG;
  }
  const int n = B * (dim / 2);
  launch_dependent(sinusoidal_kernel, (n + 127) / 128, 128, 0, stream, t, out, B, dim);
  return after_launch("sinusoidal_kernel");
}

int launch_pos_table(float* table, int h, int w, int E, int pmax, int base_size,
                     cudaStream_t stream) {
  if (!table || h <= 0 || w <= 0 || E <= 0 || (E & 3) || h > pmax || w > pmax || base_size <= 0) {
    set_last_error("pos_table: invalid argument (grid %dx%d, max %d, E %d)", h, w, pmax, E);
    return ST_INVALID_ARG;
  }
  const long total = static_cast<long>(h) * w * (E / 4);
  pos_table_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(table, h, w, E,
                                                                                  pmax, base_size);
  return after_launch("pos_table_kernel");
}

int launch_patchify(const void* latent, int in_f32, void* out, bool out_planes, int B, int C, int H,
                    int W, int p, cudaStream_t stream) {
  if (!latent || !out || B <= 0 || C <= 0 || p <= 0 || H % p || W % p) {
    set_last_error("patchify: invalid argument");
    return ST_INVALID_ARG;
  }
  const long total = static_cast<long>(B) * C * H * W;
  const unsigned grid = static_cast<unsigned>((total + 255) / 256);
  if (in_f32 && out_planes)
    launch_dependent(patchify_kernel<float, true>, grid, 256, 0, stream, (const float*)latent, (bf16*)out, B, C, H, W, p);
  else if (out_planes)
    launch_dependent(patchify_kernel<bf16, true>, grid, 256, 0, stream, (const bf16*)latent, (bf16*)out, B, C, H, W, p);
  else if (in_f32)
    launch_dependent(patchify_kernel<float, false>, grid, 256, 0, stream, (const float*)latent, (bf16*)out, B, C, H, W, p);
  else
    launch_dependent(patchify_kernel<bf16, false>, grid, 256, 0, stream, (const bf16*)latent, (bf16*)out, B, C, H, W, p);
  return after_launch("patchify_kernel");
}

// ----------------------------------------------------------------------------
// e4m3 operands for the FP8 GEMM: out = saturate(in * inv_scale), round to
// nearest even; and the absolute maximum a scale is derived from.
// ----------------------------------------------------------------------------
namespace {

template <typename TI>
__global__ void quantize_e4m3_kernel(const TI* in, uint8_t* out, long n,
                                     float inv_scale) {
  grid_dep_wait();
  grid_dep_launch();
  // four elements per thread per step (n is a multiple of 4)
  long i = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x * 4;
  for (; i < n; i += stride) {
    float v[4];
    if constexpr (sizeof(TI) == 4) {
      const float4 f = *reinterpret_cast<const float4*>(in + i);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
      const uint2 u = *reinterpret_cast<const uint2*>(in + i);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
    const uint32_t lo = pack_e4m3x2(v[0] * inv_scale, v[1] * inv_scale);
    const uint32_t hi = pack_e4m3x2(v[2] * inv_scale, v[3] * inv_scale);
    *reinterpret_cast<uint32_t*>(out + i) = lo | (hi << 16);
  }
}

template <typename TI>
__global__ void absmax_kernel(const TI* __restrict__ in, long n, unsigned* __restrict__ out_bits) {
  float m = 0.f;
  long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x;
  for (; i < n; i += stride) {
    float v;
    if constexpr (sizeof(TI) == 4) v = in[i]; else v = __bfloat162float(in[i]);
    m = fmaxf(m, fabsf(v));
  }
  m = warp_max(m);
  // non-negative floats order like their bit patterns
  if ((threadIdx.x & 31) == 0) atomicMax(out_bits, __float_as_uint(m));
}

}  // namespace

int launch_quantize_e4m3(const void* in, int in_f32, void* out, long n, float inv_scale,
                         cudaStream_t stream) {
  if (!in || !out || n <= 0 || n % 4 != 0 || (reinterpret_cast<uintptr_t>(in) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 3)) {
    set_last_error("quantize_e4m3: need n %% 4 == 0 and aligned pointers (n %ld)", n);
    return ST_INVALID_ARG;
  }
  const long blocks = (n / 4 + 255) / 256;
  const unsigned grid = static_cast<unsigned>(blocks < device_sm_count() * 16 ? blocks : device_sm_count() * 16);
  if (in_f32)
    launch_dependent(quantize_e4m3_kernel<float>, grid, 256, 0, stream, static_cast<const float*>(in),
                                                          static_cast<uint8_t*>(out), n, inv_scale);
  else
    launch_dependent(quantize_e4m3_kernel<bf16>, grid, 256, 0, stream, static_cast<const bf16*>(in),
                                                         static_cast<uint8_t*>(out), n, inv_scale);
  return after_launch("quantize_e4m3_kernel");
}

int launch_absmax(const void* in, int in_f32, long n, float* out, cudaStream_t stream) {
  if (!in || !out || n <= 0) {
    set_last_error("absmax: invalid argument");
    return ST_INVALID_ARG;
  }
  cudaError_t e = cudaMemsetAsync(out, 0, 4, stream);
  if (e != cudaSuccess) return check_cuda(e, "cudaMemsetAsync(absmax)");
  const long blocks = (n + 255) / 256;
  const unsigned grid = static_cast<unsigned>(blocks < device_sm_count() * 8 ? blocks : device_sm_count() * 8);
  if (in_f32)
    absmax_kernel<float><<<grid, 256, 0, stream>>>(static_cast<const float*>(in), n,
                                                   reinterpret_cast<unsigned*>(out));
  else
    absmax_kernel<bf16><<<grid, 256, 0, stream>>>(static_cast<const bf16*>(in), n,
                                                  reinterpret_cast<unsigned*>(out));
  return after_launch("absmax_kernel");
}

int launch_cast_f32_to_bf16(const float* in, bf16* out, long n, cudaStream_t stream) {
  if (n <= 0) return ST_OK;
  const unsigned grid = static_cast<unsigned>(n / 256 + 1 < device_sm_count() * 16 ? n / 256 + 1 : device_sm_count() * 16);
  launch_dependent(cast_kernel<float, bf16>, grid, 256, 0, stream, in, out, n);
  return after_launch("cast_kernel");
}

int launch_cast_bf16_to_f32(const bf16* in, float* out, long n, cudaStream_t stream) {
  if (n <= 0) return ST_OK;
  const unsigned grid = static_cast<unsigned>(n / 256 + 1 < device_sm_count() * 16 ? n / 256 + 1 : device_sm_count() * 16);
  launch_dependent(cast_kernel<bf16, float>, grid, 256, 0, stream, in, out, n);
  return after_launch("cast_kernel");
}

int launch_transpose(const void* in, int in_f32, void* out, int out_f32, int R, int C,
                     cudaStream_t stream) {
  if (!in || !out || R <= 0 || C <= 0) {
    set_last_error("transpose: invalid argument");
    return ST_INVALID_ARG;
  }
  const dim3 grid((C + 31) / 32, (R + 31) / 32), block(32, 8);
  if (in_f32 && out_f32)
    transpose_kernel<float, float><<<grid, block, 0, stream>>>((const float*)in, (float*)out, R, C);
  else if (in_f32)
    transpose_kernel<float, bf16><<<grid, block, 0, stream>>>((const float*)in, (bf16*)out, R, C);
  else if (out_f32)
    transpose_kernel<bf16, float><<<grid, block, 0, stream>>>((const bf16*)in, (float*)out, R, C);
  else
    transpose_kernel<bf16, bf16><<<grid, block, 0, stream>>>((const bf16*)in, (bf16*)out, R, C);
  return after_launch("transpose_kernel");
}

int launch_split3(const void* in, int in_f32, bf16* out, long n, cudaStream_t stream) {
  if (!in || !out || n <= 0 || n % 4 || (reinterpret_cast<uintptr_t>(out) & 7)) {
    set_last_error("split3: need n %% 4 == 0 and an aligned output (n %ld)", n);
    return ST_INVALID_ARG;
  }
  const bool vec = (reinterpret_cast<uintptr_t>(in) & (in_f32 ? 15 : 7)) == 0;
  const long blocks = (n / 4 + 255) / 256, most = device_sm_count() * 16L;
  const unsigned grid = static_cast<unsigned>(blocks < most ? blocks : most);
  if (in_f32)
    launch_dependent(vec ? split3_kernel<float, true> : split3_kernel<float, false>, grid, 256, 0, stream,
                     static_cast<const float*>(in), out, n);
  else
    launch_dependent(vec ? split3_kernel<bf16, true> : split3_kernel<bf16, false>, grid, 256, 0, stream,
                     static_cast<const bf16*>(in), out, n);
  return after_launch("split3_kernel");
}

int launch_transpose_split3(const void* in, int in_f32, bf16* out, int R, int C, cudaStream_t stream) {
  if (!in || !out || R <= 0 || C <= 0 || R % 2 || (static_cast<long>(R) * C) % 2) {
    set_last_error("transpose_split3: invalid argument (R %d must be even)", R);
    return ST_INVALID_ARG;
  }
  const dim3 grid((C + 31) / 32, (R + 63) / 64), block(32, 8);
  if (in_f32)
    transpose_split3_kernel<float><<<grid, block, 0, stream>>>(static_cast<const float*>(in), out, R, C);
  else
    transpose_split3_kernel<bf16><<<grid, block, 0, stream>>>(static_cast<const bf16*>(in), out, R, C);
  return after_launch("transpose_split3_kernel");
}

int launch_rmsnorm_heads(void* x, int x_f32, long ld, long rows, int col0, int nheads, int D,
                         const float* w, float eps, cudaStream_t stream) {
  if (!x || rows <= 0 || nheads <= 0 || D <= 0) {
    set_last_error("rmsnorm_heads: invalid argument");
    return ST_INVALID_ARG;
  }
  const long units = rows * nheads;
  const unsigned grid = static_cast<unsigned>((units + 7) / 8);
  if (x_f32)
    launch_dependent(rmsnorm_heads_kernel<float>, grid, 256, 0, stream, (float*)x, ld, rows, col0, nheads, D, w, eps);
  else
    launch_dependent(rmsnorm_heads_kernel<bf16>, grid, 256, 0, stream, (bf16*)x, ld, rows, col0, nheads, D, w, eps);
  return after_launch("rmsnorm_heads_kernel");
}


// ----------------------------------------------------------------------------
// Generic 2-D convolution (any square stride and zero padding), one thread per
// output element, fp32 accumulation.  Off the denoiser's path (its patch
// embedding is kernel == stride and runs as a gather + tensor-core GEMM); this
// is the stand-alone `conv2d` operator of the reference (conv2d,
// modules.cpp:1037-1062) for the shapes its own script uses.
// ----------------------------------------------------------------------------
namespace {
template <typename T>
__global__ void conv2d_direct_kernel(const T* __restrict__ in, const float* __restrict__ w,
                                     const float* __restrict__ bias, T* __restrict__ out, int B, int C, int H,
                                     int W, int O, int kh, int kw, int stride, int pad, int Ho, int Wo) {
  const long total = static_cast<long>(B) * O * Ho * Wo;
  for (long idx = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long>(gridDim.x) * blockDim.x) {
    const int xo = static_cast<int>(idx % Wo);
    const int yo = static_cast<int>((idx / Wo) % Ho);
    const int o = static_cast<int>((idx / (static_cast<long>(Wo) * Ho)) % O);
    const int b = static_cast<int>(idx / (static_cast<long>(Wo) * Ho * O));
    float acc = bias ? bias[o] : 0.f;
    for (int c = 0; c < C; ++c) {
      const T* ip = in + (static_cast<long>(b) * C + c) * H * W;
      const float* wp = w + (static_cast<long>(o) * C + c) * kh * kw;
      for (int ky = 0; ky < kh; ++ky) {
        const int y = yo * stride - pad + ky;
        if (y < 0 || y >= H) continue;
        for (int kx = 0; kx < kw; ++kx) {
          const int x = xo * stride - pad + kx;
          if (x < 0 || x >= W) continue;
          float v;
          if constexpr (sizeof(T) == 4) v = ip[static_cast<long>(y) * W + x];
          else v = __bfloat162float(ip[static_cast<long>(y) * W + x]);
          acc = fmaf(v, wp[ky * kw + kx], acc);
        }
      }
    }
    if constexpr (sizeof(T) == 4) out[idx] = acc;
    else out[idx] = __float2bfloat16(acc);
  }
}
}  // namespace

int launch_conv2d_direct(const void* in, int io_f32, const float* w, const float* bias, void* out, int B, int C,
                         int H, int W, int O, int kh, int kw, int stride, int pad, cudaStream_t stream) {
  if (!in || !w || !out || B <= 0 || C <= 0 || H <= 0 || W <= 0 || O <= 0 || kh <= 0 || kw <= 0 || stride <= 0 ||
      pad < 0 || H + 2 * pad < kh || W + 2 * pad < kw) {
    set_last_error("conv2d: invalid argument");
    return ST_INVALID_ARG;
  }
  const int Ho = (H + 2 * pad - kh) / stride + 1, Wo = (W + 2 * pad - kw) / stride + 1;
  const long total = static_cast<long>(B) * O * Ho * Wo;
  const long blocks = (total + 255) / 256;
  const unsigned grid = static_cast<unsigned>(blocks < device_sm_count() * 16L ? blocks : device_sm_count() * 16L);
  if (io_f32)
    conv2d_direct_kernel<float><<<grid, 256, 0, stream>>>(static_cast<const float*>(in), w, bias,
                                                          static_cast<float*>(out), B, C, H, W, O, kh, kw, stride,
                                                          pad, Ho, Wo);
  else
    conv2d_direct_kernel<bf16><<<grid, 256, 0, stream>>>(static_cast<const bf16*>(in), w, bias,
                                                         static_cast<bf16*>(out), B, C, H, W, O, kh, kw, stride, pad,
                                                         Ho, Wo);
  return after_launch("conv2d_direct_kernel");
}

}  // namespace sd3
