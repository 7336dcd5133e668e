// Multi-adapter LoRA on the token stream of one engine step: y[t] += B_s (A_s x[t]) with s = the adapter slot of token t.
//
// Reference seam: /root/reference/src/vllm_tgis_adapter/grpc/adapters.py:63-163 turns a request's adapter_id into a
// `lora_request=LoRARequest(...)` kwarg of engine.generate (grpc_server.py:205-225); the arithmetic is vLLM's:
//   vllm/lora/layers/base_linear.py `apply`            y = base_layer(x); punica.add_lora_linear(y, x, A, B, scale=1.0)
//   vllm/lora/punica_wrapper/punica_gpu.py             buffer = zeros(fp32); add_shrink(buffer, x, A, scale);
//                                                      add_expand(y, buffer, B, add_inputs=True)
//   vllm/lora/ops/triton_ops/lora_shrink_op.py         fp32 accumulation of x . A^T, stored to the fp32 buffer
//   vllm/lora/ops/triton_ops/lora_expand_op.py         buffer cast to the weight dtype (bf16), fp32 accumulation of
//                                                      buffer . B^T, result cast to bf16, then y = y + result (bf16 add)
//   vllm/lora/lora_weights.py `optimize`               the alpha/r scaling is folded into B once at load time (host side)
// Rounding points restated here exactly: fp32 shrink sums -> bf16 -> fp32 expand sums -> bf16 delta -> bf16(y + delta).
//
// Shape of the problem: HBM/L2-bound skinny products (rank 8..64 against K, N of 1k..14k), integer slot look-ups per
// token; no tensor-core shape worth having.  Two kernels per adapted projection group:
//   shrink : CTA = (tile of 8 tokens, 4 rank rows of one module), its 8 warps split K; the A rows are streamed once per
//            tile and adapter with 16-byte loads and used for all of the tile's tokens of that adapter.
//   expand : CTA = (tile of 8 tokens, 1024 output columns), thread = 4 consecutive columns; the 4 B rows of a thread are
//            one contiguous run (a warp reads 32 consecutive runs -- fully coalesced) and are read ONCE for the tile's tokens
//            of one adapter; the tile's rank vectors are staged in shared memory (broadcast reads).
// Both are launches of a few microseconds of dependent loads.  The engine runs shrink BEFORE the base projection, which it
// does not depend on: the projection's first weights are on their way while it runs.
// Adapter storage (engine.cu): per layer and module  A [slots][Rm][K] and B [slots][N][Rm] bf16, zero padded to the module's
// rank capacity Rm, so no kernel needs the adapter's true rank.  gate_proj / up_proj are stored as ONE module of capacity
// 2R over the interleaved gate_up projection (row 2j = gate_j, row 2j+1 = up_j: block-sparse B), see engine.cu.
#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace tgis {

namespace {

// 8 consecutive bf16 values as fp32 through ONE 16-byte load (an aggregate of eight __nv_bfloat16 read element-wise compiles
// to eight 2-byte loads: the first version of these kernels ran 10x slower for exactly that reason)
struct F8 {
  float v[8];
};
__device__ __forceinline__ float dot8(const F8& a, const F8& b) {
  float s = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) s = fmaf(a.v[e], b.v[e], s);
  return s;
}

constexpr int LORA_TT = 8;  // tokens per tile
constexpr int LORA_MAX_RM = 128;

// The adapter slots of a tile's tokens (-1 behind the last token).  A tile is worked through once per distinct slot -- the
// scheduler sorts a step's tokens by adapter, so most tiles have one or two --, by different CTAs in small launches.
struct TileSlots {
  int s[LORA_TT];
  __device__ __forceinline__ TileSlots(const int32_t* tok_slot, int t0, int T) {
#pragma unroll
    for (int j = 0; j < LORA_TT; ++j) s[j] = t0 + j < T ? tok_slot[t0 + j] : -1;
  }
  // the p-th distinct slot from `least` on, in the order of first tokens; -1: there are fewer
  __device__ __forceinline__ int distinct(int p, int least) const {
    int found = -1, n = 0;
#pragma unroll
    for (int j = 0; j < LORA_TT; ++j) {
      bool first = s[j] >= least;
#pragma unroll
      for (int i = 0; i < j; ++i) first &= s[i] != s[j];
      if (first && n++ == p) found = s[j];
    }
    return found;
  }
};
inline int lora_passes_apart(int T) { return T <= 1 ? 1 : T <= 256 ? 4 : 1; }   // CTAs that share a tile's distinct slots

__device__ __forceinline__ F8 cvt8(const uint4& r) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
  F8 o;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    o.v[2 * e] = __uint_as_float(w[e] << 16);
    o.v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
  }
  return o;
}

// shrink: CTA = (tile of 8 tokens, LORA_RPC = 4 rank rows of one module); its 8 warps split K (warp w owns the 16-byte
// vectors w*32 + lane + 256 i), so a decode-shaped launch is 16 .. 50 CTAs of two to seven dependent load rounds each
// instead of a handful of warps walking a whole row (the first version: 16 .. 56 serial memory latencies per launch), and
// the tile's x vectors are loaded once for the four rows (one row per CTA made a prefill chunk L2-bandwidth bound:
// 16 CTAs re-read the same 64 KB of x).  Partial sums meet in shared memory and are added in warp order: deterministic.
constexpr int LORA_RPC = 4;
__global__ void __launch_bounds__(256)
lora_shrink_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const int32_t* __restrict__ tok_slot, LoraGroup g,
                   float* __restrict__ v, int T) {
  __shared__ float part[8][LORA_RPC][LORA_TT];
  griddep_launch();
  griddep_wait();
  int m = 0, r0 = (int)blockIdx.y * LORA_RPC;  // blockIdx.y enumerates (module, group of LORA_RPC rank rows)
  while (m + 1 < g.n_mods && r0 >= g.mod[m].Rm) {
    r0 -= g.mod[m].Rm;
    ++m;
  }
  const LoraModule md = g.mod[m];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = (int)blockIdx.x * LORA_TT;
  const TileSlots tile(tok_slot, t0, T);
  const int nvec = md.K / 8;
  const uint4* xq = reinterpret_cast<const uint4*>(x);
  const size_t ldq = (size_t)ldx / 8;
  for (int p = blockIdx.z;; p += gridDim.z) {
    const int slot = tile.distinct(p, 1);
    if (slot < 0) return;
    float acc[LORA_RPC][LORA_TT];
#pragma unroll
    for (int q = 0; q < LORA_RPC; ++q)
#pragma unroll
      for (int j = 0; j < LORA_TT; ++j) acc[q][j] = 0.f;
    const uint4* a0 = reinterpret_cast<const uint4*>(md.A + ((size_t)(slot - 1) * md.Rm + r0) * md.K);
    for (int kv = warp * 32 + lane; kv < nvec; kv += 256) {
      uint4 ar[LORA_RPC], xr[LORA_TT];
#pragma unroll
      for (int q = 0; q < LORA_RPC; ++q) ar[q] = a0[(size_t)q * nvec + kv];
#pragma unroll
      for (int j = 0; j < LORA_TT; ++j) xr[j] = tile.s[j] == slot ? xq[(size_t)(t0 + j) * ldq + kv] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int j = 0; j < LORA_TT; ++j) {
        const F8 xf = cvt8(xr[j]);
#pragma unroll
        for (int q = 0; q < LORA_RPC; ++q) acc[q][j] += dot8(cvt8(ar[q]), xf);
      }
    }
#pragma unroll
    for (int q = 0; q < LORA_RPC; ++q)
#pragma unroll
      for (int j = 0; j < LORA_TT; ++j) {
        float s = acc[q][j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) part[warp][q][j] = s;
      }
    __syncthreads();
    if (threadIdx.x < LORA_RPC * LORA_TT) {
      const int q = threadIdx.x / LORA_TT, j = threadIdx.x % LORA_TT;
      if (t0 + j < T && tok_slot[t0 + j] == slot) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += part[w][q][j];
        v[(size_t)(t0 + j) * g.v_ld + md.v_off + r0 + q] = s;
      }
    }
    __syncthreads();   // part is used again
  }
}

// expand: CTA = (tile of 8 tokens, 1024 output columns), thread = LORA_EC = 4 consecutive columns (~100 registers: two
// CTAs per SM).  Same-adapter tile: per 8 rank indices the thread holds its 4 x 8 block of B in registers -- the next
// block is already in flight while this one is used -- and, per rank index, the tile's 8 rank values arrive as two
// broadcast 16-byte shared-memory loads (32 FMAs per 2 LDS; the first version paid one LDS per FMA and one exposed memory
// latency per block).
constexpr int LORA_EC = 4;
constexpr int LORA_ECOLS = 256 * LORA_EC;  // columns per CTA
__device__ __forceinline__ void st4f(__nv_bfloat16* p, const float (&f)[4]) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(f[0], f[1]), hi = __floats2bfloat162_rn(f[2], f[3]);
  uint2 r;
  r.x = *reinterpret_cast<const uint32_t*>(&lo);
  r.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = r;
}
// ACT: the columns are interleaved (gate_j, up_j) pairs; act[t, j] = bf16(silu(gate)) * up of the corrected projection is
// written (for tokens without an adapter too) and y is only read: the projection's own kernel after it drops out.
template <bool ACT>
__global__ void __launch_bounds__(256)
lora_expand_kernel(const float* __restrict__ v, const int32_t* __restrict__ tok_slot, LoraGroup g,
                   __nv_bfloat16* __restrict__ y, int ldy, __nv_bfloat16* __restrict__ act, int T) {
  __shared__ __align__(16) float vsT[LORA_MAX_RM][LORA_TT];  // [rank index][token of the tile]
  griddep_launch();
  griddep_wait();
  const int t0 = (int)blockIdx.y * LORA_TT;
  const LoraModule md = g.mod[blockIdx.z % g.n_mods];
  if ((int)blockIdx.x * LORA_ECOLS >= md.N) return;
  const TileSlots tile(tok_slot, t0, T);
  const int n0 = ((int)blockIdx.x * 256 + (int)threadIdx.x) * LORA_EC;
  const bool col_ok = n0 < md.N;
  for (int p = blockIdx.z / g.n_mods;; p += gridDim.z / g.n_mods) {
    const int slot = tile.distinct(p, ACT ? 0 : 1);
    if (slot < 0) return;
    // the thread's y values and its first block of B do not depend on the rank vectors -- request them before the staging
    // barrier so that their latency runs under it (a CTA is only a few microseconds of work)
    uint2 yraw[LORA_TT];
    uint4 nxt[LORA_EC];
    const __nv_bfloat16* brow = md.B + ((size_t)(slot > 0 ? slot - 1 : 0) * md.N + (col_ok ? n0 : 0)) * md.Rm;
    if (col_ok) {
      if (slot > 0) {
#pragma unroll
        for (int e = 0; e < LORA_EC; ++e) nxt[e] = *reinterpret_cast<const uint4*>(brow + (size_t)e * md.Rm);
      }
#pragma unroll
      for (int j = 0; j < LORA_TT; ++j)
        if (tile.s[j] == slot) yraw[j] = *reinterpret_cast<const uint2*>(y + (size_t)(t0 + j) * ldy + md.col0 + n0);
    }
    float acc[LORA_TT][LORA_EC];
#pragma unroll
    for (int j = 0; j < LORA_TT; ++j)
#pragma unroll
      for (int e = 0; e < LORA_EC; ++e) acc[j][e] = 0.f;
    if (slot > 0) {
      // the fp32 shrink sums enter the second product as bf16 (lora_expand_op.py casts the buffer to the weight dtype)
      for (int i = threadIdx.x; i < LORA_TT * md.Rm; i += 256) {
        const int j = i / md.Rm, r = i - j * md.Rm;
        const bool live = t0 + j < T && tok_slot[t0 + j] == slot;
        vsT[r][j] = live ? bf16_round(v[(size_t)(t0 + j) * g.v_ld + md.v_off + r]) : 0.f;
      }
      __syncthreads();
      if (col_ok) {
        const int nrv = md.Rm / 8;
        for (int rv = 0; rv < nrv; ++rv) {
          F8 bb[LORA_EC];
#pragma unroll
          for (int e = 0; e < LORA_EC; ++e) bb[e] = cvt8(nxt[e]);
          if (rv + 1 < nrv) {
#pragma unroll
            for (int e = 0; e < LORA_EC; ++e) nxt[e] = *reinterpret_cast<const uint4*>(brow + (size_t)e * md.Rm + 8 * (rv + 1));
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 va = *reinterpret_cast<const float4*>(&vsT[rv * 8 + q][0]);
            const float4 vb = *reinterpret_cast<const float4*>(&vsT[rv * 8 + q][4]);
            const float vv[LORA_TT] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
#pragma unroll
            for (int e = 0; e < LORA_EC; ++e)
#pragma unroll
              for (int j = 0; j < LORA_TT; ++j) acc[j][e] = fmaf(vv[j], bb[e].v[q], acc[j][e]);
          }
        }
      }
    }
    if (col_ok) {
#pragma unroll
      for (int j = 0; j < LORA_TT; ++j) {
        if (tile.s[j] != slot) continue;   // (another adapter's token: its sums here are not used)
        float yv[LORA_EC] = {__uint_as_float(yraw[j].x << 16), __uint_as_float(yraw[j].x & 0xffff0000u),
                             __uint_as_float(yraw[j].y << 16), __uint_as_float(yraw[j].y & 0xffff0000u)};
        if (slot > 0) {
#pragma unroll
          for (int e = 0; e < LORA_EC; ++e) yv[e] += bf16_round(acc[j][e]);
        }
        if constexpr (ACT) {
          float o[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float gx = bf16_round(yv[2 * h]);
            o[h] = bf16_round(gx / (1.0f + expf(-gx))) * bf16_round(yv[2 * h + 1]);
          }
          *reinterpret_cast<__nv_bfloat162*>(act + (size_t)(t0 + j) * (md.N / 2) + n0 / 2) = __floats2bfloat162_rn(o[0], o[1]);
        } else {
          st4f(y + (size_t)(t0 + j) * ldy + md.col0 + n0, yv);
        }
      }
    }
    __syncthreads();   // vsT is used again
  }
}

}  // namespace

static bool lora_group_ok(const LoraGroup& g) {
  if (g.n_mods < 1 || g.n_mods > LORA_GROUP_MAX) return false;
  for (int m = 0; m < g.n_mods; ++m) {
    const LoraModule& md = g.mod[m];
    if (md.Rm < 8 || md.Rm > LORA_MAX_RM || md.Rm % 8 != 0 || md.K % 8 != 0 || md.N % 8 != 0 || md.col0 % 8 != 0) return false;
  }
  return true;
}

cudaError_t lora_shrink_launch(const __nv_bfloat16* x, int ldx, const int32_t* tok_slot, const LoraGroup& g, float* v, int T,
                               cudaStream_t stream) {
  if (T <= 0) return cudaSuccess;
  if (!lora_group_ok(g) || ldx % 8 != 0) return cudaErrorInvalidValue;
  int groups = 0;
  for (int m = 0; m < g.n_mods; ++m) groups += g.mod[m].Rm / LORA_RPC;
  return launch_k(lora_shrink_kernel, dim3((T + LORA_TT - 1) / LORA_TT, groups, lora_passes_apart(T)), dim3(256), 0, stream, x, ldx, tok_slot,
                  g, v, T);
}

cudaError_t lora_expand_launch(const float* v, const int32_t* tok_slot, const LoraGroup& g, __nv_bfloat16* y, int ldy, int T,
                               cudaStream_t stream, __nv_bfloat16* act) {
  if (T <= 0) return cudaSuccess;
  if (!lora_group_ok(g) || ldy % 8 != 0 || (act != nullptr && (g.n_mods != 1 || g.mod[0].col0 != 0))) return cudaErrorInvalidValue;
  int max_n = 0;
  for (int m = 0; m < g.n_mods; ++m) max_n = g.mod[m].N > max_n ? g.mod[m].N : max_n;
  const dim3 grid((max_n + LORA_ECOLS - 1) / LORA_ECOLS, (T + LORA_TT - 1) / LORA_TT, g.n_mods * lora_passes_apart(T));
  return act != nullptr ? launch_k(lora_expand_kernel<true>, grid, dim3(256), 0, stream, v, tok_slot, g, y, ldy, act, T)
                        : launch_k(lora_expand_kernel<false>, grid, dim3(256), 0, stream, v, tok_slot, g, y, ldy, act, T);
}

}  // namespace tgis
