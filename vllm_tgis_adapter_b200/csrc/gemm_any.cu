// General matrix product  Y = X W^T  for the shapes the tcgen05 kernel does not take: any T / N / K and leading
// dimensions, bf16 or fp32 operands (fp32 accumulation in both cases; fp32 operands are multiplied in true fp32, no TF32),
// three launch geometries
//   dense    one problem,
//   batched  blockIdx.z walks equal problems whose operands lie a fixed stride apart (one problem per attention head),
//   grouped  the rows are cut into segments (seg_off, on the device) and segment g multiplies with weight matrix g
//            (one segment per expert of a mixture-of-experts layer); rows of X may be gathered through an index list,
// and seven epilogues (plain store, SwiGLU or GeGLU over interleaved gate/up rows, per-(row, batch) scale, tanh, squared ReLU of
// the row-scaled sum, exact gelu).
//
// Every output element is a sum in an order of k that only K and the kernel fix, so a row's result depends neither on the
// other rows of the launch nor on where in a segment it landed.
//
// Kernels: grouped bf16 products run on CTA pairs where their rows allow it (gemm_pair.cu); a handful of outputs over long
// rows (router and gate projections of a decode step) take one warp per output (gemm_any_rowdot_kernel); bf16 operands whose
// rows start on 16-byte boundaries run on the tensor cores (gemm_any_mma_kernel); everything else -- fp32 operands, odd
// leading dimensions -- runs on the FMA pipe (gemm_any_kernel).  Dense launches that fit the tcgen05 kernels' operand layout
// are routed there by the engine.
#include <cstdint>
#include <cstdlib>

#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace tgis {
namespace {

constexpr int ANY_THREADS = 256;

template <class T>
__device__ __forceinline__ float ld_as_float(const T* p);
template <>
__device__ __forceinline__ float ld_as_float<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float ld_as_float<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void st_from_float(float* p, float v) { *p = v; }
__device__ __forceinline__ void st_from_float(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
// act(gate) * up: silu (GEMM_ANY_SWIGLU) or the tanh form of gelu (GEMM_ANY_GEGLU)
__device__ __forceinline__ float glu_pair(int mode, float g, float u) {
  if (mode == GEMM_ANY_SWIGLU) return g / (1.f + expf(-g)) * u;
  return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
}

__device__ __forceinline__ float gelu_erf(float z) { return 0.5f * z * (1.f + erff(z * 0.7071067811865476f)); }
// max(acc * s, 0)^2 with s the scale of the row's INPUT (GEMM_ANY_RELU2)
__device__ __forceinline__ float relu2_scaled(float acc, float s) {
  const float z = fmaxf(acc * s, 0.f);
  return z * z;
}
__device__ __forceinline__ float relu2_row_scale(const GemmAny& a, int dst) {
  return a.row_scale == nullptr ? 1.f : a.row_scale[a.gather != nullptr ? a.gather[dst] : dst];
}

// ---- FMA pipe: fp32 operands (true fp32), fp32 activations under bf16 weights, odd leading dimensions -----------------
// CTA tile BM x 64 of 128 threads (8 x 16), a thread owns rows ty + 8 i and columns tx + 16 j.  Bound by the FMA pipe: operands
// are kept in shared memory as they lie in memory ([row][k], rows padded to 36 floats so that eight neighbouring rows start
// in different bank groups), a thread reads four k of a row with one 16-byte load, and both halves of a packed
// multiply-add take neighbouring k: an output is the sum over even k plus the sum over odd k, each in ascending order, which
// no other row and no tile height enters.  BM / 8 + 4 loads feed BM packed multiply-adds of two k each.  The next k-block's
// global loads (16 bytes each where the rows allow it) are in flight while this one is worked on.
// Measured, fp32, T x N x K (before: scalar staging, one 16-byte and several 4-byte shared loads for 16 multiply-adds, nothing
// in flight; then with half-warps instead of neighbouring lanes on one weight row): 389 x 1088 x 1024 149 -> 47 -> 41 us, 16 experts of
// 2048 x 1024 under 778 rows 296 -> 165 (tiles of 64 rows) -> 118 us, 10 x 32768 x 1024 189 -> 57 -> 44 us.  With one or two warps to a
// scheduler the waits between dependent instructions are what is left; the operands of the next four k in registers ahead: no faster (41).
constexpr int FMA_THREADS = 128;
constexpr int FMA_BN = 64, FMA_BK = 32, FMA_LD = FMA_BK + 4;
constexpr int FMA_SMS = 148;   // (tile heights only: a sum does not depend on them)
// Sums of up to 64 terms run as one ascending chain per output, not as an even and an odd one that meet at the end.  The reason is
// which values they give, not speed: small float32 models are compared with 64-bit arithmetic to within 1e-4, some of them are
// conditioned so badly that one ulp of the inputs moves their logits by as much, and this is the order in which they were
// always summed.  Both orders are equally exact (the bound in the tests holds for either).  It costs time: 2048 x 2048 44 us at K = 64
// against 40 at K = 68 in packed pairs, 512 x 1024 8.3 against 8.1, 93 x 128 7.6 against 6.2.
constexpr int FMA_CHAIN_K = 64;

__device__ __forceinline__ void fma_low(unsigned long long& d, float x, float w) {   // the pair's lower half
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(fmaf(x, w, lo)), "f"(hi));
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long x, unsigned long long y) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(d) : "l"(x), "l"(y));
}
__device__ __forceinline__ float sum2(unsigned long long v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
template <bool VEC>
__device__ __forceinline__ float4 ld4(const float* p, int left) {   // `left` elements of the row from p on
  if constexpr (VEC) return left > 0 ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
}
template <bool VEC>
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p, int left) {
  if constexpr (VEC) {
    if (left <= 0) return make_float4(0.f, 0.f, 0.f, 0.f);
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
  }
  return make_float4(left > 0 ? __bfloat162float(p[0]) : 0.f, left > 1 ? __bfloat162float(p[1]) : 0.f, left > 2 ? __bfloat162float(p[2]) : 0.f,
                     left > 3 ? __bfloat162float(p[3]) : 0.f);
}

template <class XT, class WT, class OT, int BM, bool VEC>
__global__ void __launch_bounds__(FMA_THREADS) gemm_any_kernel(GemmAny a) {
  constexpr int TM = BM / 8, TN = FMA_BN / 16;
  constexpr int XV = BM * FMA_BK / 4 / FMA_THREADS, WV = FMA_BN * FMA_BK / 4 / FMA_THREADS;   // 4-element pieces a thread stages
  __shared__ __align__(16) float Xs[2][BM * FMA_LD];
  __shared__ __align__(16) float Ws[2][FMA_BN * FMA_LD];
  __shared__ int row_src[BM], row_dst[BM];
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x;
  // ---- which rows
  int row0, row_end, group = 0;
  if (a.seg_off != nullptr) {
    int t = blockIdx.y;
    for (; group < a.n_groups; ++group) {
      const int cnt = a.seg_off[group + 1] - a.seg_off[group];
      const int nt = (cnt + BM - 1) / BM;
      if (t < nt) break;
      t -= nt;
    }
    if (group >= a.n_groups) return;
    row0 = a.seg_off[group] + t * BM;
    row_end = a.seg_off[group + 1];
  } else {
    row0 = blockIdx.y * BM;
    row_end = a.T;
  }
  if (tid < BM) {
    const int r = row0 + tid;
    int src = -1;
    if (r < row_end) src = a.gather != nullptr ? a.gather[r] / a.gather_div : r;
    row_src[tid] = src;
    row_dst[tid] = r < row_end ? r : -1;
  }
  __syncthreads();
  const int z = blockIdx.z;
  const XT* X = reinterpret_cast<const XT*>(a.X) + (size_t)z * a.x_bs;
  const WT* W = reinterpret_cast<const WT*>(a.W) + (size_t)z * a.w_bs + (size_t)group * a.w_gs;
  OT* Y = reinterpret_cast<OT*>(a.Y) + (size_t)z * a.y_bs;
  const int n0 = blockIdx.x * FMA_BN;
  // neighbouring lanes share a weight row: a 16-byte load whose lanes agree in pairs takes two passes over the banks, one whose half-warps
  // agree takes four
  const int ty = tid / 32 * 2 + (tid & 1), tx = tid % 32 / 2;

  // pieces of four k: piece e -> row e / 8, k 4 (e % 8)
  const int pk = (tid & 7) * 4, pr = tid >> 3;
  const XT* xp[XV];
  const WT* wp[WV];
#pragma unroll
  for (int i = 0; i < XV; ++i) {
    const int src = row_src[pr + i * (FMA_THREADS / 8)];
    xp[i] = src >= 0 ? X + (size_t)src * a.ldx + pk : nullptr;
  }
#pragma unroll
  for (int i = 0; i < WV; ++i) {
    const int n = n0 + pr + i * (FMA_THREADS / 8);
    wp[i] = n < a.N ? W + (size_t)n * a.ldw + pk : nullptr;
  }
  float4 xv[XV], wv[WV];
  auto fetch = [&](int k0) {
    const int left = a.K - k0 - pk;
#pragma unroll
    for (int i = 0; i < XV; ++i) xv[i] = ld4<VEC>(xp[i] + k0, xp[i] != nullptr ? left : 0);
#pragma unroll
    for (int i = 0; i < WV; ++i) wv[i] = ld4<VEC>(wp[i] + k0, wp[i] != nullptr ? left : 0);
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int i = 0; i < XV; ++i) *reinterpret_cast<float4*>(&Xs[buf][(pr + i * (FMA_THREADS / 8)) * FMA_LD + pk]) = xv[i];
#pragma unroll
    for (int i = 0; i < WV; ++i) *reinterpret_cast<float4*>(&Ws[buf][(pr + i * (FMA_THREADS / 8)) * FMA_LD + pk]) = wv[i];
  };
  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  fetch(0);
  put(0);
  __syncthreads();
  const int KB = (a.K + FMA_BK - 1) / FMA_BK;
  for (int kb = 0; kb < KB; ++kb) {
    const int cur = kb & 1;
    if (kb + 1 < KB) fetch((kb + 1) * FMA_BK);
    const float* xs = &Xs[cur][ty * FMA_LD];
    const float* ws = &Ws[cur][tx * FMA_LD];
    if (a.K <= FMA_CHAIN_K) {
#pragma unroll 1
      for (int k = 0; k < FMA_BK; ++k) {
        float w1[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) w1[j] = ws[j * 16 * FMA_LD + k];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) fma_low(acc[i][j], xs[i * 8 * FMA_LD + k], w1[j]);
      }
    } else
#pragma unroll
    for (int k = 0; k < FMA_BK; k += 4) {
      ulonglong2 w2[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w2[j] = *reinterpret_cast<const ulonglong2*>(ws + j * 16 * FMA_LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(xs + i * 8 * FMA_LD + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          fma2(acc[i][j], x2.x, w2[j].x);
          fma2(acc[i][j], x2.y, w2[j].y);
        }
      }
    }
    if (kb + 1 < KB) {
      put(cur ^ 1);   // (last read two k-blocks ago, before the barrier below)
      __syncthreads();
    }
  }
  // ---- epilogue: a thread's columns are 16 apart; gate and up of a pair sit two threads apart
  const bool glu = a.mode == GEMM_ANY_SWIGLU || a.mode == GEMM_ANY_GEGLU;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int dst = row_dst[ty + 8 * i];
    const float s = dst < 0 ? 1.f : a.mode == GEMM_ANY_ROWSCALE ? a.row_scale[(size_t)dst * a.scale_ld + z] : a.mode == GEMM_ANY_RELU2 ? relu2_row_scale(a, dst) : 1.f;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 16 * j;
      const float v = sum2(acc[i][j]);
      if (glu) {   // columns (2c, 2c + 1) = (gate_c, up_c): out[c] = act(gate) * up
        const float up = __shfl_down_sync(0xffffffffu, v, 2);
        if ((tx & 1) == 0 && dst >= 0 && n + 1 < a.N) st_from_float(Y + (size_t)dst * a.ldy + n / 2, glu_pair(a.mode, v, up));
      } else if (dst >= 0 && n < a.N) {
        const float o = a.mode == GEMM_ANY_RELU2 ? relu2_scaled(v, s) : a.mode == GEMM_ANY_TANH ? tanhf(v) : a.mode == GEMM_ANY_GELU ? gelu_erf(v) : v * s;
        st_from_float(Y + (size_t)dst * a.ldy + n, o);
      }
    }
  }
}

// ---- tensor-core variant (bf16 operands, 16-byte aligned rows): mma.sync m16n8k16, fp32 accumulators ---------------
// CTA tile 64 or 128 rows x 128 weight rows, k-blocks of 32 in a three-stage cp.async ring (out-of-range rows and the k tail
// are zero-filled by the copy), 8 warps as 2 x 4; operands reach the registers through ldmatrix from rows
// padded to 80 bytes (conflict-free).  Same geometries and epilogues as the FMA kernel; the k order inside an output
// element is fixed (ascending k-blocks, the MMA's own order inside), so a row's result does not depend on its neighbours.
constexpr int MMA_BN = 128, MMA_BK = 32, MMA_LD = MMA_BK + 8;

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem, bool valid) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* smem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}

// MI = 16-row MMA tiles per warp along M: CTA tile (32 MI) rows x 128 weight rows (MI = 2: 64 rows, MI = 4: 128 rows).
// Dynamic shared memory: MMA_STAGES x (32 MI + 128) rows of MMA_LD bf16.
constexpr int MMA_STAGES = 3;
template <int MI>
constexpr size_t mma_smem_bytes() { return (size_t)MMA_STAGES * (32 * MI + MMA_BN) * MMA_LD * 2; }

template <class OT, int MI>
__global__ void __launch_bounds__(ANY_THREADS) gemm_any_mma_kernel(GemmAny a) {
  using bf = __nv_bfloat16;
  constexpr int BM = 32 * MI;
  extern __shared__ __align__(16) unsigned char mma_smem[];
  bf* Xs = reinterpret_cast<bf*>(mma_smem);                 // [stage][BM][MMA_LD]
  bf* Ws = Xs + (size_t)MMA_STAGES * BM * MMA_LD;           // [stage][MMA_BN][MMA_LD]
  __shared__ int row_src[BM], row_dst[BM];
  griddep_launch();
  griddep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int row0, row_end, group = 0;
  if (a.seg_off != nullptr) {
    int t = blockIdx.y;
    for (; group < a.n_groups; ++group) {
      const int cnt = a.seg_off[group + 1] - a.seg_off[group];
      const int nt = (cnt + BM - 1) / BM;
      if (t < nt) break;
      t -= nt;
    }
    if (group >= a.n_groups) return;
    row0 = a.seg_off[group] + t * BM;
    row_end = a.seg_off[group + 1];
  } else {
    row0 = blockIdx.y * BM;
    row_end = a.T;
  }
  if (tid < BM) {
    const int r = row0 + tid;
    row_src[tid] = r < row_end ? (a.gather != nullptr ? a.gather[r] / a.gather_div : r) : -1;
    row_dst[tid] = r < row_end ? r : -1;
  }
  __syncthreads();
  const int z = blockIdx.z;
  const bf* X = reinterpret_cast<const bf*>(a.X) + (size_t)z * a.x_bs;
  const bf* W = reinterpret_cast<const bf*>(a.W) + (size_t)z * a.w_bs + (size_t)group * a.w_gs;
  OT* Y = reinterpret_cast<OT*>(a.Y) + (size_t)z * a.y_bs;
  const int n0 = blockIdx.x * MMA_BN;
  const int wm = warp >> 2, wn = warp & 3;  // 2 x 4 warps, warp tile (16 MI) x 32

  auto stage_load = [&](int st, int k0) {
    bf* xs = Xs + (size_t)st * BM * MMA_LD;
    bf* ws = Ws + (size_t)st * MMA_BN * MMA_LD;
#pragma unroll
    for (int i = 0; i < BM / 64; ++i) {  // X: BM rows x 4 chunks of 8 elements
      const int id = tid + i * ANY_THREADS;
      const int r = id >> 2, c = id & 3;
      const int src = row_src[r];
      const bool ok = src >= 0 && k0 + c * 8 < a.K;
      cp_async_16(xs + (size_t)r * MMA_LD + c * 8, ok ? X + (size_t)src * a.ldx + k0 + c * 8 : X, ok);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {  // W: 128 rows x 4 chunks
      const int id = tid + i * ANY_THREADS;
      const int n = id >> 2, c = id & 3;
      const bool ok = n0 + n < a.N && k0 + c * 8 < a.K;
      cp_async_16(ws + (size_t)n * MMA_LD + c * 8, ok ? W + (size_t)(n0 + n) * a.ldw + k0 + c * 8 : W, ok);
    }
  };

  float acc[MI][4][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

  const int KB = (a.K + MMA_BK - 1) / MMA_BK;
#pragma unroll
  for (int s = 0; s < MMA_STAGES - 1; ++s) {  // prologue (one commit group per stage, empty ones included)
    if (s < KB) stage_load(s, s * MMA_BK);
    cp_async_commit();
  }
  for (int kb = 0; kb < KB; ++kb) {
    cp_async_wait<MMA_STAGES - 2>();  // k-block kb has landed (for this thread's copies)
    __syncthreads();                  // ... for everyone's; and everyone is done with the stage refilled below
    if (kb + MMA_STAGES - 1 < KB) stage_load((kb + MMA_STAGES - 1) % MMA_STAGES, (kb + MMA_STAGES - 1) * MMA_BK);
    cp_async_commit();
    const bf* xs = Xs + (size_t)(kb % MMA_STAGES) * BM * MMA_LD;
    const bf* ws = Ws + (size_t)(kb % MMA_STAGES) * MMA_BN * MMA_LD;
#pragma unroll
    for (int ks = 0; ks < MMA_BK / 16; ++ks) {
      uint32_t af[MI][4], bfr[2][4];
#pragma unroll
      for (int mi = 0; mi < MI; ++mi)
        ldsm_x4(af[mi], xs + (size_t)(wm * 16 * MI + mi * 16 + (lane & 15)) * MMA_LD + ks * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int nj = 0; nj < 2; ++nj)
        ldsm_x4(bfr[nj], ws + (size_t)(wn * 32 + nj * 16 + (lane >> 4) * 8 + (lane & 7)) * MMA_LD + ks * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) mma_16816(acc[mi][ni], af[mi], bfr[ni >> 1][(ni & 1) * 2], bfr[ni >> 1][(ni & 1) * 2 + 1]);
    }
  }
  // ---- epilogue: a thread holds columns (2t, 2t + 1) of rows g and g + 8 of every 16 x 8 block
  const int g = lane >> 2, t2 = (lane & 3) * 2;
#pragma unroll
  for (int mi = 0; mi < MI; ++mi)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int dst = row_dst[wm * 16 * MI + mi * 16 + g + half * 8];
      if (dst < 0) continue;
      const float s = a.mode == GEMM_ANY_ROWSCALE ? a.row_scale[(size_t)dst * a.scale_ld + z]
                      : a.mode == GEMM_ANY_RELU2  ? relu2_row_scale(a, dst) : 1.f;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int n = n0 + wn * 32 + ni * 8 + t2;
        const float v0 = acc[mi][ni][half * 2], v1 = acc[mi][ni][half * 2 + 1];
        if (a.mode == GEMM_ANY_SWIGLU || a.mode == GEMM_ANY_GEGLU) {
          if (n + 1 < a.N) st_from_float(Y + (size_t)dst * a.ldy + n / 2, glu_pair(a.mode, v0, v1));
        } else if (a.mode == GEMM_ANY_TANH) {
          if (n < a.N) st_from_float(Y + (size_t)dst * a.ldy + n, tanhf(v0));
          if (n + 1 < a.N) st_from_float(Y + (size_t)dst * a.ldy + n + 1, tanhf(v1));
        } else if (a.mode == GEMM_ANY_GELU) {
          if (n < a.N) st_from_float(Y + (size_t)dst * a.ldy + n, gelu_erf(v0));
          if (n + 1 < a.N) st_from_float(Y + (size_t)dst * a.ldy + n + 1, gelu_erf(v1));
        } else if (a.mode == GEMM_ANY_RELU2) {
          if (n < a.N) st_from_float(Y + (size_t)dst * a.ldy + n, relu2_scaled(v0, s));
          if (n + 1 < a.N) st_from_float(Y + (size_t)dst * a.ldy + n + 1, relu2_scaled(v1, s));
        } else {
          if (n < a.N) st_from_float(Y + (size_t)dst * a.ldy + n, v0 * s);
          if (n + 1 < a.N) st_from_float(Y + (size_t)dst * a.ldy + n + 1, v1 * s);
        }
      }
    }
}

template <class OT, int MI>
cudaError_t launch_mma_mi(const GemmAny& a, cudaStream_t stream) {
  constexpr int BM = 32 * MI;
  static bool attr_set = false;
  if (!attr_set) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_any_mma_kernel<OT, MI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)mma_smem_bytes<MI>());
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  const int row_tiles = a.seg_off != nullptr ? (a.T + BM - 1) / BM + a.n_groups : (a.T + BM - 1) / BM;
  const dim3 grid((a.N + MMA_BN - 1) / MMA_BN, row_tiles, a.batch > 0 ? a.batch : 1);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
  return launch_k(gemm_any_mma_kernel<OT, MI>, grid, dim3(ANY_THREADS), mma_smem_bytes<MI>(), stream, a);
}

template <class OT>
cudaError_t launch_mma(const GemmAny& a, cudaStream_t stream) {
  // 128-row tiles once the problems (or the average expert segment) are tall enough to fill them
  const int rows = a.seg_off != nullptr ? (a.T + a.n_groups - 1) / (a.n_groups > 0 ? a.n_groups : 1) : a.T;
  return rows > 96 ? launch_mma_mi<OT, 4>(a, stream) : launch_mma_mi<OT, 2>(a, stream);
}

bool mma_eligible(const GemmAny& a) {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("TGIS_GEMM_ANY_MMA");
    on = (e && e[0] == '0') ? 0 : 1;
  }
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return on && a.x_dtype == DT_BF16 && a.w_dtype == DT_BF16 && a.K % 8 == 0 && a.ldx % 8 == 0 && a.ldw % 8 == 0 &&
         a.x_bs % 8 == 0 && a.w_bs % 8 == 0 && a.w_gs % 8 == 0 && al16(a.X) && al16(a.W);
}

// ---- few outputs, long rows (a router or gate projection in a decode step): one warp per output element -------------
// lanes stride the reduction (coalesced), fixed shuffle tree at the end; any alignment, any operand types.
template <class XT, class WT, bool VEC8>
__global__ void __launch_bounds__(ANY_THREADS) gemm_any_rowdot_kernel(GemmAny a) {
  griddep_launch();
  griddep_wait();
  const int lane = threadIdx.x & 31;
  const long long out = (long long)blockIdx.x * (ANY_THREADS / 32) + (threadIdx.x >> 5);
  if (out >= (long long)a.T * a.N) return;
  const int t = (int)(out / a.N), n = (int)(out % a.N);
  const XT* x = reinterpret_cast<const XT*>(a.X) + (size_t)t * a.ldx;
  const WT* w = reinterpret_cast<const WT*>(a.W) + (size_t)n * a.ldw;
  float acc = 0.f;
  if (VEC8) {  // bf16 rows on 16-byte boundaries, K % 8 == 0: 8 elements per load, several loads in flight
    const uint4* x4 = reinterpret_cast<const uint4*>(x);
    const uint4* w4 = reinterpret_cast<const uint4*>(w);
#pragma unroll 8
    for (int c = lane; c < a.K / 8; c += 32) {
      const uint4 xv = x4[c], wv = w4[c];
      const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&xv);
      const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&wv);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 xf = __bfloat1622float2(xp[e]), wf = __bfloat1622float2(wp[e]);
        acc = fmaf(xf.x, wf.x, acc);
        acc = fmaf(xf.y, wf.y, acc);
      }
    }
  } else {
#pragma unroll 4
    for (int k = lane; k < a.K; k += 32) acc = fmaf(ld_as_float(x + k), ld_as_float(w + k), acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) {
    if (a.mode == GEMM_ANY_TANH) acc = tanhf(acc);
    if (a.y_dtype == DT_BF16) reinterpret_cast<__nv_bfloat16*>(a.Y)[(size_t)t * a.ldy + n] = __float2bfloat16_rn(acc);
    else reinterpret_cast<float*>(a.Y)[(size_t)t * a.ldy + n] = acc;
  }
}
bool rowdot_eligible(const GemmAny& a) {
  // With a tanh (the low-rank decay map) the line lies in tokens alone, where other products change their kernel too.  bf16, K = 2048,
  // microseconds, tiles of the mma.sync kernel -> here, 32, 64, 128 and 256 tokens: 64 outputs 32 35 53 53 -> 2.9 3.9 5.6 9.5, 127 outputs 32 37
  // 55 55 -> 4.0 5.7 9.5 17.0; K = 4096, 64 outputs: 58 66 92 92 -> 4.0 5.8 8.5 14.9.  (More tokens: gemm_pair_takes_dense.)
  const bool bf16 = a.x_dtype == DT_BF16 && a.w_dtype == DT_BF16;
  const bool few = a.mode == GEMM_ANY_TANH ? a.T <= (bf16 ? 256 : 64) : a.mode == GEMM_ANY_PLAIN && a.y_dtype == DT_F32 && (long long)a.T * a.N <= 8192;
  return a.seg_off == nullptr && a.batch <= 1 && few && a.N < 128 && a.K >= 256 && !(a.x_dtype == DT_BF16 && a.w_dtype == DT_F32);
}
template <class XT, class WT, bool VEC8 = false>
cudaError_t launch_rowdot(const GemmAny& a, cudaStream_t stream) {
  const long long outs = (long long)a.T * a.N;
  return launch_k(gemm_any_rowdot_kernel<XT, WT, VEC8>, dim3((unsigned)((outs + ANY_THREADS / 32 - 1) / (ANY_THREADS / 32))),
                  dim3(ANY_THREADS), 0, stream, a);
}

template <class XT, class WT, class OT, int BM>
cudaError_t launch_fma_bm(const GemmAny& a, bool vec, cudaStream_t stream) {
  const int row_tiles = a.seg_off != nullptr ? (a.T + BM - 1) / BM + a.n_groups : (a.T + BM - 1) / BM;
  const dim3 grid((a.N + FMA_BN - 1) / FMA_BN, row_tiles, a.batch > 0 ? a.batch : 1);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
  return vec ? launch_k(gemm_any_kernel<XT, WT, OT, BM, true>, grid, dim3(FMA_THREADS), 0, stream, a)
             : launch_k(gemm_any_kernel<XT, WT, OT, BM, false>, grid, dim3(FMA_THREADS), 0, stream, a);
}
template <class XT, class WT, class OT>
cudaError_t launch_fma(const GemmAny& a, cudaStream_t stream) {
  // four elements per load: rows, problems and segments start on a multiple of four elements' bytes, K is a multiple of four
  auto al = [](const void* p, size_t esz) { return (reinterpret_cast<uintptr_t>(p) & (4 * esz - 1)) == 0; };
  const bool vec = a.K % 4 == 0 && a.ldx % 4 == 0 && a.ldw % 4 == 0 && a.x_bs % 4 == 0 && a.w_bs % 4 == 0 && a.w_gs % 4 == 0 &&
                   al(a.X, sizeof(XT)) && al(a.W, sizeof(WT));
  // rows per tile: 16 for skinny problems (decode steps, small segments); 64 where that makes three tiles for every SM, else 32
  // (K = 1024: 389 x 2048 57 us with 32 rows, 66 with 64; 2048 x 4096 478 and 431).  Segments take 32: they end inside their last tile
  // (16 experts of 2048 x 1024, 16 / 32 / 64 rows: 389 rows in all 82 / 74 / 127, 778 129 / 118 / 130, 4096 549 / 472 / 500)
  const int rows = a.seg_off != nullptr ? (a.T + a.n_groups - 1) / (a.n_groups > 0 ? a.n_groups : 1) : a.T;
  const long long tiles64 = (long long)((a.N + FMA_BN - 1) / FMA_BN) * (a.batch > 0 ? a.batch : 1) * ((a.T + 63) / 64);
  // (16 rows too where 32 would leave half of the SMs without a tile and K is short: 32 x 4096 x 128 13.6 -> 7.4 us)
  const long long tiles32 = (long long)((a.N + FMA_BN - 1) / FMA_BN) * (a.batch > 0 ? a.batch : 1) * ((rows + 31) / 32);
  if (rows <= 20 || (a.seg_off == nullptr && a.K <= 256 && 2 * tiles32 <= FMA_SMS)) return launch_fma_bm<XT, WT, OT, 16>(a, vec, stream);
  const bool fit32 = (a.T + 31ll) / 32 + (a.seg_off != nullptr ? a.n_groups : 0) <= 65535;   // tiles of one launch (grid.y)
  if (fit32 && (a.seg_off != nullptr || rows <= 36 || tiles64 < 3 * FMA_SMS || a.K <= 256)) return launch_fma_bm<XT, WT, OT, 32>(a, vec, stream);
  return launch_fma_bm<XT, WT, OT, 64>(a, vec, stream);
}

}  // namespace

cudaError_t gemm_any_launch(const GemmAny& a, cudaStream_t stream) {
  if (a.T <= 0 || a.N <= 0) return cudaSuccess;
  if (a.K <= 0 || ((a.mode == GEMM_ANY_SWIGLU || a.mode == GEMM_ANY_GEGLU) && (a.N & 1))) return cudaErrorInvalidValue;
  if (a.mode == GEMM_ANY_ROWSCALE && a.row_scale == nullptr) return cudaErrorInvalidValue;
  if (a.gather != nullptr && a.gather_div <= 0) return cudaErrorInvalidValue;
  using bf = __nv_bfloat16;
  if (rowdot_eligible(a)) {
    if (a.x_dtype == DT_BF16) {
      const bool vec = a.K % 8 == 0 && a.ldx % 8 == 0 && a.ldw % 8 == 0 && (reinterpret_cast<uintptr_t>(a.X) & 15) == 0 &&
                       (reinterpret_cast<uintptr_t>(a.W) & 15) == 0;
      return vec ? launch_rowdot<bf, bf, true>(a, stream) : launch_rowdot<bf, bf>(a, stream);
    }
    return a.w_dtype == DT_BF16 ? launch_rowdot<float, bf>(a, stream) : launch_rowdot<float, float>(a, stream);
  }
  // expert segments: CTA pairs.  64 experts of 2 x 1408 x 2048 and back, top 6, both products in microseconds, mma.sync -> pairs:
  // 4 tokens 126 -> 78, 32 tokens 260 -> 165 (6.3 TB/s of weights), 512 tokens 334 -> 195, 2048 tokens 1003 -> 243
  if (gemm_pair_takes_groups(a)) return gemm_pair_grouped_launch(a, stream);
  if (mma_eligible(a) && gemm_pair_takes_dense(a)) return gemm_pair_dense_launch(a, stream);
  if (mma_eligible(a) && gemm_skinny_takes_batch(a)) return gemm_skinny_batch_launch(a, stream);
  if (mma_eligible(a)) return a.y_dtype == DT_BF16 ? launch_mma<bf>(a, stream) : launch_mma<float>(a, stream);
  const int key = a.x_dtype * 4 + a.w_dtype * 2 + a.y_dtype;  // DT_F32 = 0, DT_BF16 = 1
  switch (key) {
    case 0: return launch_fma<float, float, float>(a, stream);
    case 2: return launch_fma<float, bf, float>(a, stream);
    case 3: return launch_fma<float, bf, bf>(a, stream);
    case 6: return launch_fma<bf, bf, float>(a, stream);
    case 7: return launch_fma<bf, bf, bf>(a, stream);
    default: return cudaErrorInvalidValue;  // (fp32 weights under bf16 activations are not a combination any model uses)
  }
}

}  // namespace tgis
