// Y[T, N] = X[T, K] W[N, K]^T for the few tokens of a decode step (T <= 32, bf16, K a multiple of 64).
//
// Such a product is bound by its weight bytes, and below some 30 MB by what a launch takes beside them: the tcgen05 kernel
// (gemm_tcgen05.cu) sets up tensor memory and barriers, waits for TMA and reduces its k-splits across a cluster, 7 us before
// the first 4 MB.  Here a warp loads weights straight into the A fragments of mma.sync (16-byte loads; a lane's eight
// neighbouring k feed two MMAs, the k order inside a chunk of 64 being permuted alike in both operands), the warps of a CTA
// split K, and one pass through shared memory adds their sums in warp order.  Weights of the first chunk are requested before
// the previous kernel has ended, all of the CTA's weights are asked into L2.  With many weight bytes or many tokens the
// activations, which every CTA reads again, cost more than that saves; gemm_skinny_takes draws the line.
//
// Measured, microseconds with cold weights, N x K, tcgen05 -> here: 1 token 768 x 768 7.0 -> 2.7, 2048 x 2048 8.7 -> 4.0,
// 4096 x 4096 12.6 -> 8.6; 32 tokens 768 x 768 8.1 -> 3.6, 2048 x 2048 9.8 -> 5.4 (6144 x 4096 17.7 -> 20.1).
#include <type_traits>

#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace tgis {
namespace {

struct SkinnyArgs {
  const __nv_bfloat16* X; const __nv_bfloat16* W; void* Y;
  int ldy, T, N, K, mode;   // mode: the out modes of gemm_bf16_launch
  GemmRope rope;            // positions == nullptr: none
};
// The problems of blockIdx.y side by side.  A type of its own: as members of SkinnyArgs, zero for one problem, these cost every launch of
// a chain 0.13 us (768 x 768, one token 3.24 -> 3.37; a request on a 12-layer model 4.43 -> 4.53 ms).
struct SkinnyBatch : SkinnyArgs {
  int ldx;
  long long x_bs, w_bs, y_bs;    // elements between the problems
  const float* row_scale;        // modes 0 and 1: result times row_scale[token * scale_ld + problem] (nullptr: 1)
  int scale_ld;
};

// Y goes into the residual stream, resid[t] = bf16(bf16(Y[t]) + resid[t]), and every eight columns of it leave the sum of their squares:
// the number with which a thread of rmsnorm_kernel enters its reduction.
struct SkinnyAdd : SkinnyArgs {
  __nv_bfloat16* resid;
  float* ssq;                    // [T][N / 8]
};
// X is the residual stream; what is multiplied is its RMS norm, which every CTA makes from those sums in the order of rmsnorm_kernel: the
// same bits as with a launch of its own.
struct SkinnyNorm : SkinnyArgs {
  const float* ssq;              // [T][K / 8]
  const __nv_bfloat16* w_norm;
  float eps;
};

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float skinny_glu(int mode, float g, float u) {
  if (mode == 2) {   // rounding points of the unfused path
    g = bf16_round(g);
    return bf16_round(g / (1.f + expf(-g))) * bf16_round(u);
  }
  return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
}

// MT: 16-row weight tiles per CTA, NT: 8-token tiles, WARPS: k-splits (warp w takes the chunks w, w + WARPS, ...).
// ROPE (MT = 2): the CTA's two tiles are the dims [16 q, 16 q + 16) of one head and their rotary partners, 64 dims on.
template <int MT, int NT, int WARPS, bool ROPE, class Args>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 16 ? 1 : 2) gemm_skinny_kernel(const Args a) {
  constexpr bool BATCH = std::is_same<Args, SkinnyBatch>::value, ADD = std::is_same<Args, SkinnyAdd>::value, NORM = std::is_same<Args, SkinnyNorm>::value;
  static_assert(!(ADD || NORM) || (NT == 1 && WARPS >= 8), "a warp per token makes its norm");
  constexpr int R = 16 * MT, TT = 8 * NT, LD = R + 1;
  extern __shared__ __align__(16) float part[];   // [WARPS][TT][LD]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = ROPE ? (blockIdx.x >> 2) * HEAD_DIM + (blockIdx.x & 3) * 16 : blockIdx.x * R;
  constexpr int M_STEP = ROPE ? 64 : 16;
  const __nv_bfloat16 *X = a.X, *W = a.W;
  int ldx = a.K;
  if constexpr (BATCH) {
    X += (size_t)blockIdx.y * a.x_bs;
    W += (size_t)blockIdx.y * a.w_bs;
    ldx = a.ldx;
  }
  if (threadIdx.x < MT) {   // weights are static: the CTA's rows (one run of bytes per tile) start on their way to L2
    const int row = n0 + (int)threadIdx.x * M_STEP, bytes = min(16, a.N - row) * a.K * 2;
    const char* from = reinterpret_cast<const char*>(W + (size_t)row * a.K);
    for (int off = 0; off < bytes; off += 65536)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(from + off), "r"(min(bytes - off, 65536)) : "memory");
  }
  griddep_launch();
  const int chunks = a.K / 64;
  const __nv_bfloat16* wr[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) wr[m][h] = W + (size_t)min(n0 + m * M_STEP + h * 8 + g, a.N - 1) * a.K + t * 8;
  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) xr[n] = X + (size_t)min(n * 8 + g, a.T - 1) * ldx + t * 8;
  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
  uint4 wv[MT][2][2];   // the next chunk
  auto load_w = [&](int c) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int s = 0; s < 2; ++s) wv[m][h][s] = ldg_stream(wr[m][h] + c * 64 + s * 32);
  };
  if (warp < chunks) load_w(warp);   // (weights are static)
  uint4 nw[2], x0[2];                // NORM: the norm's weights of a chunk, the first chunk of X
  float rs = 0.f;                    // ... and 1 / rms of the lane's token
  if constexpr (NORM) {
#pragma unroll
    for (int s = 0; s < 2; ++s) nw[s] = warp < chunks ? *reinterpret_cast<const uint4*>(a.w_norm + warp * 64 + s * 32 + t * 8) : make_uint4(0, 0, 0, 0);
  }
  griddep_wait();
  if constexpr (NORM) {
    __shared__ float rs_s[8];
#pragma unroll
    for (int s = 0; s < 2; ++s) x0[s] = warp < chunks ? *reinterpret_cast<const uint4*>(xr[0] + warp * 64 + s * 32) : make_uint4(0, 0, 0, 0);
    if (warp < a.T) {
      const int np = a.K / 8;
      float v[8], tot = 0.f;   // 256 threads of eight columns: eight warps' sums, then theirs
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = q * 32 + lane < np ? a.ssq[(size_t)warp * np + q * 32 + lane] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
#pragma unroll
      for (int q = 0; q < 8; ++q) tot = lane == q ? v[q] : tot;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
      if (lane == 0) rs_s[warp] = rsqrtf(tot / (float)a.K + a.eps);
    }
    __syncthreads();
    rs = rs_s[min(g, a.T - 1)];
  }
  for (int c = warp; c < chunks; c += WARPS) {
    uint4 xv[NT][2], wc[MT][2][2];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if constexpr (NORM) {
          if (c != warp) {
            x0[s] = *reinterpret_cast<const uint4*>(xr[n] + c * 64 + s * 32);
            nw[s] = *reinterpret_cast<const uint4*>(a.w_norm + c * 64 + s * 32 + t * 8);
          }
          const uint32_t xs[4] = {x0[s].x, x0[s].y, x0[s].z, x0[s].w}, ws[4] = {nw[s].x, nw[s].y, nw[s].z, nw[s].w};
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float lo = bf16_round(__uint_as_float(xs[e] << 16) * rs) * __uint_as_float(ws[e] << 16);
            const float hi = bf16_round(__uint_as_float(xs[e] & 0xffff0000u) * rs) * __uint_as_float(ws[e] & 0xffff0000u);
            const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
            o[e] = *reinterpret_cast<const uint32_t*>(&p);
          }
          xv[n][s] = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
          xv[n][s] = *reinterpret_cast<const uint4*>(xr[n] + c * 64 + s * 32);
        }
      }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int s = 0; s < 2; ++s) wc[m][h][s] = wv[m][h][s];
    if (c + WARPS < chunks) load_w(c + WARPS);
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          mma_16816(acc[m][n], wc[m][0][s].x, wc[m][1][s].x, wc[m][0][s].y, wc[m][1][s].y, xv[n][s].x, xv[n][s].y);
          mma_16816(acc[m][n], wc[m][0][s].z, wc[m][1][s].z, wc[m][0][s].w, wc[m][1][s].w, xv[n][s].z, xv[n][s].w);
        }
  }
  // acc[m][n]: rows g, g + 8 of weight tile m, tokens 2t, 2t + 1 of token tile n
  float* mine = part + (size_t)warp * TT * LD;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) mine[(n * 8 + 2 * t + (e & 1)) * LD + m * 16 + g + (e >> 1) * 8] = acc[m][n][e];
  __syncthreads();
  auto sum = [&](int tok, int j) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) v += part[((size_t)w * TT + tok) * LD + j];
    return v;
  };
  __nv_bfloat16* __restrict__ Y = reinterpret_cast<__nv_bfloat16*>(a.Y);
  if constexpr (ADD) {
    for (int i = threadIdx.x; i < ((a.T * R + 31) & ~31); i += WARPS * 32) {   // (whole warps: eight lanes meet)
      const int tok = i / R, j = i % R;
      const bool in = tok < a.T && n0 + j < a.N;
      __nv_bfloat16* r = a.resid + (size_t)tok * a.N + n0 + j;
      float z = 0.f;
      if (in) {
        const __nv_bfloat16 v = __float2bfloat16_rn(bf16_round(sum(tok, j)) + __bfloat162float(*r));
        *r = v;
        z = __bfloat162float(v);
      }
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float f = __shfl_sync(0xffffffffu, z, (lane & ~7) + e);
        ss = fmaf(f, f, ss);
      }
      if (in && (j & 7) == 0) a.ssq[(size_t)tok * (a.N / 8) + (n0 + j) / 8] = ss;
    }
  } else if constexpr (ROPE) {
    // rotary embedding and the scatter into the paged cache (arithmetic and rounding points of rope_kvwrite_kernel)
    const int head = n0 / HEAD_DIM, d0 = n0 % HEAD_DIM;
    for (int i = threadIdx.x; i < a.T * 16; i += WARPS * 32) {
      const int tok = i >> 4, j = i & 15, d = d0 + j;
      float lo = bf16_round(sum(tok, j)), hi = bf16_round(sum(tok, 16 + j));
      if (head < a.rope.n_q + a.rope.n_kv) {
        const __nv_bfloat16* cs = a.rope.cos_sin + (size_t)a.rope.positions[tok] * HEAD_DIM + d;
        const float c = __bfloat162float(cs[0]), s = __bfloat162float(cs[64]), l = lo, h = hi;
        lo = bf16_round(l * c) - bf16_round(h * s);
        hi = bf16_round(h * c) + bf16_round(l * s);
      }
      const __nv_bfloat16 out[2] = {__float2bfloat16_rn(lo), __float2bfloat16_rn(hi)};
      __nv_bfloat16* y = Y + (size_t)tok * a.ldy + n0 + j;
      y[0] = out[0];
      y[64] = out[1];
      const int slot = head >= a.rope.n_q ? a.rope.slot_mapping[tok] : -1;
      if (slot >= 0) {
        const int blk = slot / KV_BLOCK, off = slot % KV_BLOCK;
        const bool key = head < a.rope.n_q + a.rope.n_kv;
        __nv_bfloat16* base = (key ? a.rope.k_cache : a.rope.v_cache) +
                              ((size_t)blk * a.rope.n_kv + (head - a.rope.n_q - (key ? 0 : a.rope.n_kv))) * (KV_BLOCK * HEAD_DIM);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const int dim = d + 64 * p, chunk = dim >> 3, sub = dim & 7;
          base[key ? (chunk * KV_BLOCK + off) * 8 + sub : off * HEAD_DIM + ((chunk ^ (off & 7)) * 8) + sub] = out[p];
        }
      }
    }
  } else if (a.mode == 2 || a.mode == 3) {   // rows (2j, 2j + 1) of W are (gate_j, up_j)
    for (int i = threadIdx.x; i < a.T * (R / 2); i += WARPS * 32) {
      const int tok = i / (R / 2), j = i % (R / 2);
      if (n0 + 2 * j + 1 < a.N) Y[(size_t)tok * a.ldy + n0 / 2 + j] = __float2bfloat16_rn(skinny_glu(a.mode, sum(tok, 2 * j), sum(tok, 2 * j + 1)));
    }
  } else {
    for (int i = threadIdx.x; i < a.T * R; i += WARPS * 32) {
      const int tok = i / R, j = i % R;
      if (n0 + j >= a.N) continue;
      float v = sum(tok, j);
      size_t o = (size_t)tok * a.ldy + n0 + j;
      if constexpr (BATCH) {
        if (a.row_scale != nullptr) v *= a.row_scale[(size_t)tok * a.scale_ld + blockIdx.y];
        o += (size_t)blockIdx.y * a.y_bs;
      }
      if (a.mode == 1) {
        reinterpret_cast<float*>(a.Y)[o] = v;
      } else {
        if (a.mode == 4) {
          v = fmaxf(v, 0.f);
          v *= v;
        }
        Y[o] = __float2bfloat16_rn(v);
      }
    }
  }
}

template <int MT, int NT, int WARPS, bool ROPE, class Args>
cudaError_t launch(const Args& a, cudaStream_t s, int problems = 1) {
  constexpr size_t smem = (size_t)WARPS * 8 * NT * (16 * MT + 1) * sizeof(float);
  static const cudaError_t attr =
      cudaFuncSetAttribute(gemm_skinny_kernel<MT, NT, WARPS, ROPE, Args>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (attr != cudaSuccess) return attr;
  return launch_k(gemm_skinny_kernel<MT, NT, WARPS, ROPE, Args>, dim3((a.N + 16 * MT - 1) / (16 * MT), problems), dim3(WARPS * 32), smem, s, a);
}
template <int MT, int WARPS, bool ROPE, class Args>
cudaError_t launch_nt(const Args& a, cudaStream_t s, int problems = 1) {
  switch ((a.T + 7) / 8) {
    case 1: return launch<MT, 1, WARPS, ROPE>(a, s, problems);
    case 2: return launch<MT, 2, WARPS, ROPE>(a, s, problems);
    case 3: return launch<MT, 3, WARPS, ROPE>(a, s, problems);
    default: return launch<MT, 4, WARPS, ROPE>(a, s, problems);
  }
}

constexpr int SKINNY_ONE_WAVE = 148 * 16;   // weight rows that 16-row CTAs cover with one CTA per SM (a constant: bits hang on it)

}  // namespace

// Where the line lies was measured inside decode steps, where the tcgen05 kernel's ring (19 MB over all SMs) fills while the
// kernel before it still runs.  Up to eight tokens: weights of up to 34 MB (steps of an 8B layer: o projection of 34 MB 1.5 %
// faster, qkv of 50 MB and more slower; steps of a 2048-wide expert model 8 to 11 % faster).  Up to 32 tokens: 9 MB (steps of
// a 2048-wide recurrent model 6 % faster at 32 tokens; an expert model with products of 9.4 MB 1 % slower).
bool gemm_skinny_takes(int T, int N, int K) {
  return T >= 1 && T <= 32 && K >= 64 && K % 64 == 0 && N <= 24576 && (long long)N * K <= (T <= 8 ? 17000000 : 4500000);
}

cudaError_t gemm_skinny_launch(const void* X, const void* W, void* Y, int ldy, int T, int N, int K, int out_mode, const GemmRope* rope,
                               cudaStream_t stream) {
  SkinnyArgs a{(const __nv_bfloat16*)X, (const __nv_bfloat16*)W, Y, ldy, T, N, K, out_mode, {}};
  // The number of warps, and with it the order of k, hangs on N alone: a row has the same bits beside 31 others as alone, and with
  // every epilogue.  Sixteen warps where an SM holds one CTA, of 16 rows up to one wave, of 32 rows up to two; eight beyond that,
  // with 32-row CTAs for few tokens (more loads in flight) and 16-row ones beyond eight (fewer activation bytes in flight per
  // register).  Between one and two waves eight warps were measured too, microseconds at 1, 8, 9, 16, 24 and 32 tokens, warm
  // weights, eight warps of 16 rows -> sixteen of 32: 2560 x 1024 2.4 2.5 2.8 3.1 3.5 4.0 -> 2.2 2.2 2.5 2.6 3.5 4.4, 4608 x 960
  // 2.4 2.6 2.9 3.1 3.6 4.1 -> 2.2 2.2 2.8 2.8 3.9 4.7.
  const bool sixteen = N <= 2 * SKINNY_ONE_WAVE;
  if (rope != nullptr) {
    a.rope = *rope;
    return sixteen ? launch_nt<2, 16, true>(a, stream) : launch_nt<2, 8, true>(a, stream);
  }
  if (!sixteen) return T <= 8 ? launch<2, 1, 8, false>(a, stream) : launch_nt<1, 8, false>(a, stream);
  return N > SKINNY_ONE_WAVE ? launch_nt<2, 16, false>(a, stream) : launch_nt<1, 16, false>(a, stream);
}

// Norms between the products of a small model's decode steps, for up to eight tokens: the product in front adds to the residual stream and
// leaves sums of squares, the one behind normalises its rows as it loads them.  In a chain a launch of its own costs 0.45 us more (12
// layers 768 wide, one request, 17 + 16 tokens: 4.34 -> 4.17 ms).  Every CTA reading the whole row and norming it over again had been slower
// than that launch (6.9 us against 4.0 + 2.0): it had a row to wait for and to sum; here it has hidden / 256 numbers a lane, three at 768, at most eight.
bool gemm_skinny_norm_takes(int T, int hidden, int q_dim, int qkv_dim, int ffn) {
  return T >= 1 && T <= 8 && hidden % 8 == 0 && hidden <= 2048 &&   // (2048: one vector a thread of rmsnorm_kernel)
         gemm_skinny_takes(T, qkv_dim, hidden) && gemm_skinny_takes(T, hidden, q_dim) && gemm_skinny_takes(T, 2 * ffn, hidden) && gemm_skinny_takes(T, hidden, ffn);
}
cudaError_t gemm_skinny_add_launch(const void* X, const void* W, __nv_bfloat16* resid, float* ssq, int T, int N, int K, cudaStream_t stream) {
  if (T < 1 || T > 8 || N % 8 != 0 || N > SKINNY_ONE_WAVE || !gemm_skinny_takes(T, N, K)) return cudaErrorInvalidValue;
  const SkinnyAdd a{{(const __nv_bfloat16*)X, (const __nv_bfloat16*)W, nullptr, N, T, N, K, 0, {}}, resid, ssq};
  return launch<1, 1, 16, false>(a, stream);
}
cudaError_t gemm_skinny_norm_launch(const void* h, const float* ssq, const __nv_bfloat16* w_norm, float eps, const void* W, void* Y, int ldy, int T, int N, int K,
                                    int out_mode, const GemmRope* rope, cudaStream_t stream) {
  if (T < 1 || T > 8 || K > 2048 || !gemm_skinny_takes(T, N, K)) return cudaErrorInvalidValue;
  SkinnyNorm a{{(const __nv_bfloat16*)h, (const __nv_bfloat16*)W, Y, ldy, T, N, K, out_mode, {}}, ssq, w_norm, eps};
  const bool sixteen = N <= 2 * SKINNY_ONE_WAVE;   // (as above)
  if (rope != nullptr) {
    a.rope = *rope;
    return sixteen ? launch<2, 1, 16, true>(a, stream) : launch<2, 1, 8, true>(a, stream);
  }
  if (!sixteen) return launch<2, 1, 8, false>(a, stream);
  return N > SKINNY_ONE_WAVE ? launch<2, 1, 16, false>(a, stream) : launch<1, 1, 16, false>(a, stream);
}

// One product per head (the up-projections that latent attention folds into queries and outputs), up to 32 tokens: grid (16 weight
// rows, problem), four warps up to 256 k, eight beyond.  32 tokens, 16 heads, microseconds, mma.sync tiles of 64 x 128 -> here:
// 512 x 128 9.4 -> 4.4, 128 x 512 (16 tiles in all) 15.5 -> 3.7.
bool gemm_skinny_takes_batch(const GemmAny& a) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return a.batch > 1 && a.batch <= 65535 && a.seg_off == nullptr && a.gather == nullptr && a.x_dtype == DT_BF16 && a.w_dtype == DT_BF16 &&
         (a.mode == GEMM_ANY_PLAIN || a.mode == GEMM_ANY_ROWSCALE) && gemm_skinny_takes(a.T, a.N, a.K) &&
         (long long)a.batch * a.N * a.K <= (a.T <= 8 ? 17000000 : 4500000) && a.ldw == a.K && a.ldx >= a.K && a.ldx % 8 == 0 &&
         a.x_bs % 8 == 0 && a.w_bs % 8 == 0 && al16(a.X) && al16(a.W);
}
cudaError_t gemm_skinny_batch_launch(const GemmAny& g, cudaStream_t stream) {
  const SkinnyBatch a{{(const __nv_bfloat16*)g.X, (const __nv_bfloat16*)g.W, g.Y, g.ldy, g.T, g.N, g.K, g.y_dtype == DT_F32 ? 1 : 0, {}},
                      g.ldx, g.x_bs, g.w_bs, g.y_bs, g.mode == GEMM_ANY_ROWSCALE ? g.row_scale : nullptr, g.scale_ld};
  return g.K <= 256 ? launch_nt<1, 4, false>(a, stream, g.batch) : launch_nt<1, 8, false>(a, stream, g.batch);
}

}  // namespace tgis
