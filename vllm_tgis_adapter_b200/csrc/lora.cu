// Multi-adapter LoRA on the token stream of one engine step: y[t] += B_s (A_s x[t]) with s = the adapter slot of token t.
//
// Reference seam: src/vllm_tgis_adapter/grpc/adapters.py:63-163 turns a request's adapter_id into a
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
// Shape of the problem: skinny products (rank 8..64 against K, N of 1k..14k) of a few kilobytes to a few megabytes with integer slot
// look-ups per token.  Two kernels per adapted projection group:
//   shrink : CTA = (tile of 8 tokens, 4 rank rows of one module), its 8 warps split K; the A rows are streamed once per
//            tile and adapter with 16-byte loads and used for all of the tile's tokens of that adapter.  (As mma.sync fragments of
//            16 tokens x 16 ranks in eight parts of K a launch of a small step took 9.8 us instead of 6.6, one of 1300 tokens 74.)
//   expand : CTA = (tile of 16 tokens, 512 output columns), warp = 64 columns: B rows as fragments of mma.sync straight from global
//            memory, all requested in one round, each lane 8 neighbouring columns of 2 tokens.  24 tokens, four adapters of rank 16, 8B
//            widths, microseconds a launch against multiply-adds from shared memory (8 tokens x 1024 columns): 6.3 -> 4.0, with SwiGLU 19.8 -> 10.4.
// Both are launches of a few microseconds of dependent loads.  Shrink and the base projection read the same x and need nothing of
// each other, so shrink runs beside the projection: launched behind it, started when every block of the projection is past its own wait
// for x (griddep_launch_after; the products on tensor cores have that form), and, having done its work, it waits for the
// projection, which is what lets the expand wait for one kernel only.  Ahead of the projection it was 4 to 10 us of a chain in which
// the weights stood still (24 tokens, four adapters of rank 16, 8B widths, one layer, PDL: 144 us with shrink ahead and B asked for
// behind the expand's wait, 126 so; without adapters 102).  Where the projection runs on register products, shrink stays ahead.
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

constexpr int LORA_TT = 16;   // tokens per tile of the expand
constexpr int LORA_ST = 8;    // of the shrink
constexpr int LORA_MAX_RM = 128;

// The adapter slots of a tile's TT tokens, lane i: token i's (-1 behind the last token).  A tile is worked through once per distinct slot --
// the scheduler sorts a step's tokens by adapter, so most tiles have one or two --, by different CTAs in small launches.
template <int TT>
struct TileSlots {
  int mine;
  __device__ __forceinline__ TileSlots(const int32_t* tok_slot, int t0, int T) {
    const int i = threadIdx.x & 31;
    mine = i < TT && t0 + i < T ? tok_slot[t0 + i] : -1;
  }
  // the n-th distinct slot from `least` on, in the order of first tokens; -1: there are fewer
  __device__ __forceinline__ int distinct(int n, int least) const {
    const uint32_t same = __match_any_sync(0xffffffffu, mine);
    uint32_t firsts = __ballot_sync(0xffffffffu, mine >= least && (int)(threadIdx.x & 31) == __ffs(same) - 1);
    for (int i = 0; i < n; ++i) firsts &= firsts - 1;
    const int s = __shfl_sync(0xffffffffu, mine, firsts != 0 ? __ffs(firsts) - 1 : 0);
    return firsts != 0 ? s : -1;
  }
  __device__ __forceinline__ int of(int token) const { return __shfl_sync(0xffffffffu, mine, token); }
};
// The same for the shrink, in every thread.
struct ShrinkSlots {
  int s[LORA_ST];
  __device__ __forceinline__ ShrinkSlots(const int32_t* tok_slot, int t0, int T) {
#pragma unroll
    for (int j = 0; j < LORA_ST; ++j) s[j] = t0 + j < T ? tok_slot[t0 + j] : -1;
  }
  // the p-th distinct slot from `least` on, in the order of first tokens; -1: there are fewer
  __device__ __forceinline__ int distinct(int p, int least) const {
    int found = -1, n = 0;
#pragma unroll
    for (int j = 0; j < LORA_ST; ++j) {
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
// A launch is a chain of latencies: rows of A are asked for under the kernel before and a round ahead, 32 sums meet in 31 exchanges
// instead of 160, the modules' table is read from the parameters instead of a copy in local memory (24 requests with adapters, average
// launch, microseconds: 8.1 -> 7.3, the expands 4.8 -> 4.0 and 11.3 -> 10.4 by the last of these).
// beside: see above; x is complete when the kernel starts, so only what comes behind waits
constexpr int LORA_RPC = 4;
__global__ void __launch_bounds__(256)
lora_shrink_kernel(const __nv_bfloat16* x, int ldx, const int32_t* __restrict__ tok_slot, const __grid_constant__ LoraGroup g,
                   float* __restrict__ v, int T, int beside) {
  __shared__ float part[8][LORA_RPC][LORA_ST];
  griddep_launch();
  int m = 0, r0 = (int)blockIdx.y * LORA_RPC;  // blockIdx.y enumerates (module, group of LORA_RPC rank rows)
  while (m + 1 < g.n_mods && r0 >= g.mod[m].Rm) {
    r0 -= g.mod[m].Rm;
    ++m;
  }
  const LoraModule md = g.mod[m];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = (int)blockIdx.x * LORA_ST;
  const ShrinkSlots tile(tok_slot, t0, T);
  const int nvec = md.K / 8;
  const uint4* xq = reinterpret_cast<const uint4*>(x);
  const size_t ldq = (size_t)ldx / 8;
  bool first = true;
  for (int p = blockIdx.z;; p += gridDim.z, first = false) {
    const int slot = tile.distinct(p, 1);   // (slots and adapters are written ahead of the step: x alone is waited for)
    if (slot < 0) {
      if (first || beside) griddep_wait();   // (beside a product: the kernel behind this one waits for both by waiting for this one)
      return;
    }
    static_assert(LORA_RPC * LORA_ST == 32, "one sum per lane");
    float acc[32] = {};
    const uint4* a0 = reinterpret_cast<const uint4*>(md.A + ((size_t)(slot - 1) * md.Rm + r0) * md.K);
    uint4 ar[LORA_RPC];
    auto load_a = [&](int kv) {
#pragma unroll
      for (int q = 0; q < LORA_RPC; ++q) ar[q] = kv < nvec ? a0[(size_t)q * nvec + kv] : make_uint4(0u, 0u, 0u, 0u);
    };
    load_a(warp * 32 + lane);
    if (first && !beside) griddep_wait();
    for (int kv = warp * 32 + lane; kv < nvec; kv += 256) {
      uint4 xr[LORA_ST];
#pragma unroll
      for (int j = 0; j < LORA_ST; ++j) xr[j] = tile.s[j] == slot ? __ldcg(xq + (size_t)(t0 + j) * ldq + kv) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int j = 0; j < LORA_ST; ++j) {
        const F8 xf = cvt8(xr[j]);
#pragma unroll
        for (int q = 0; q < LORA_RPC; ++q) acc[q * LORA_ST + j] += dot8(cvt8(ar[q]), xf);
      }
      if (kv + 256 < nvec) load_a(kv + 256);
    }
    // 32 sums over 32 lanes, each lane ends with one: 31 exchanges instead of 160, the same pairs added
#pragma unroll
    for (int step = 0; step < 5; ++step) {
      const int o = 16 >> step;
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (i < o) {
          const float keep = upper ? acc[i + o] : acc[i], give = upper ? acc[i] : acc[i + o];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    part[warp][lane / LORA_ST][lane % LORA_ST] = acc[0];
    __syncthreads();
    if (threadIdx.x < LORA_RPC * LORA_ST) {
      const int q = threadIdx.x / LORA_ST, j = threadIdx.x % LORA_ST;
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

constexpr int LORA_ECOLS = 512;   // columns per CTA of the expand: 8 warps x 64
// ACT: the columns are interleaved (gate_j, up_j) pairs; act[t, j] = bf16(silu(gate)) * up of the corrected projection is
// written (for tokens without an adapter too) and y is only read: the projection's own kernel after it drops out.
// (v and y, and x of the shrink, are not __restrict__: a load through such a pointer may be moved ahead of a wait that stands in a branch)
template <bool ACT>
__global__ void __launch_bounds__(256, 2)
lora_expand_kernel(const float* v, const int32_t* __restrict__ tok_slot, const __grid_constant__ LoraGroup gr,
                   __nv_bfloat16* y, int ldy, __nv_bfloat16* __restrict__ act, int T) {
  __shared__ __align__(16) __nv_bfloat16 vs[LORA_TT][LORA_MAX_RM + 8];   // the tile's rank vectors
  griddep_launch();
  const int t0 = (int)blockIdx.y * LORA_TT;
  const LoraModule md = gr.mod[blockIdx.z % gr.n_mods];
  if ((int)blockIdx.x * LORA_ECOLS >= md.N) return;
  const TileSlots<LORA_TT> tile(tok_slot, t0, T);   // (written by the host before the step)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = (int)blockIdx.x * LORA_ECOLS + warp * 64;
  const int kc = (md.Rm + 15) / 16;   // chunks of 16 rank indices
  const int slot_of[2] = {tile.of(g), tile.of(g + 8)};
  bool first = true;
  for (int p = blockIdx.z / gr.n_mods;; p += gridDim.z / gr.n_mods) {
    const int slot = tile.distinct(p, ACT ? 0 : 1);
    if (slot < 0) {
      if (first) griddep_wait();
      return;
    }
    // the adapter's rows are static: asked for under the kernel before
    const __nv_bfloat16* brow[2][4];
    uint2 nxt[2][4];
    auto load = [&](int c) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          nxt[h][j] = c * 16 + t * 4 < md.Rm ? *reinterpret_cast<const uint2*>(brow[h][j] + c * 16 + t * 4) : make_uint2(0u, 0u);
    };
    if (slot > 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = min(n0 + 32 * h + 8 * (g >> 1) + 2 * j + (g & 1), md.N - 1);
          brow[h][j] = md.B + ((size_t)(slot - 1) * md.N + n) * md.Rm;
        }
      load(0);
    }
    if (first) griddep_wait();
    first = false;
    // columns n0 + 32 h + 8 t .. + 7 of tokens g and g + 8 are this lane's; of the products' column blocks j = 0 .. 3 (8 wide) lane
    // group t holds the neighbours 2 j, 2 j + 1, so block j is made of the columns 8 (c / 2) + 2 j + c % 2, c = 0 .. 7
    uint4 yv[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int n = n0 + 32 * h + 8 * t;
        yv[h][k] = make_uint4(0u, 0u, 0u, 0u);
        if (slot_of[k] == slot && n < md.N) {
          const uint2* from = reinterpret_cast<const uint2*>(y + (size_t)(t0 + g + 8 * k) * ldy + md.col0 + n);
          const uint2 lo = from[0], hi = from[1];
          yv[h][k] = make_uint4(lo.x, lo.y, hi.x, hi.y);
        }
      }
    float acc[2][4][4] = {};
    if (slot > 0) {
      // the fp32 shrink sums enter the second product as bf16 (lora_expand_op.py casts the buffer to the weight dtype)
      const int row4 = kc * 4;
      for (int i = threadIdx.x; i < LORA_TT * row4; i += 256) {
        const int tok = i / row4, r = i % row4 * 4;
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + tok < T && r < md.Rm && tok_slot[t0 + tok] == slot) {
          const float* from = v + (size_t)(t0 + tok) * gr.v_ld + md.v_off + r;
          f = __ldcg(reinterpret_cast<const float4*>(from));
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(f.x, f.y), hi = __floats2bfloat162_rn(f.z, f.w);
        *reinterpret_cast<uint2*>(&vs[tok][r]) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
      __syncthreads();
      for (int c = 0; c < kc; ++c) {
        uint2 bv[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 4; ++j) bv[h][j] = nxt[h][j];
        if (c + 1 < kc) load(c + 1);
        const uint2 a0 = *reinterpret_cast<const uint2*>(&vs[g][c * 16 + t * 4]), a1 = *reinterpret_cast<const uint2*>(&vs[g + 8][c * 16 + t * 4]);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 4; ++j) mma_16816(acc[h][j], a0.x, a1.x, a0.y, a1.y, bv[h][j].x, bv[h][j].y);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int n = n0 + 32 * h + 8 * t;
        if (slot_of[k] != slot || n >= md.N) continue;   // (another adapter's token: its sums here are not used)
        const uint32_t yw[4] = {yv[h][k].x, yv[h][k].y, yv[h][k].z, yv[h][k].w};
        float o[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          o[2 * j] = __uint_as_float(yw[j] << 16);
          o[2 * j + 1] = __uint_as_float(yw[j] & 0xffff0000u);
          if (slot > 0) {
            o[2 * j] += bf16_round(acc[h][j][2 * k]);
            o[2 * j + 1] += bf16_round(acc[h][j][2 * k + 1]);
          }
        }
        if constexpr (ACT) {
          float gate[4], s[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) gate[j] = bf16_round(o[2 * j]);
          silu_bf16_n(gate, s);
          const __nv_bfloat162 lo = __floats2bfloat162_rn(s[0] * bf16_round(o[1]), s[1] * bf16_round(o[3]));
          const __nv_bfloat162 hi = __floats2bfloat162_rn(s[2] * bf16_round(o[5]), s[3] * bf16_round(o[7]));
          *reinterpret_cast<uint2*>(act + (size_t)(t0 + g + 8 * k) * (md.N / 2) + n / 2) =
              make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
          uint2* to = reinterpret_cast<uint2*>(y + (size_t)(t0 + g + 8 * k) * ldy + md.col0 + n);
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 q = __floats2bfloat162_rn(o[2 * j], o[2 * j + 1]);
            w[j] = *reinterpret_cast<const uint32_t*>(&q);
          }
          to[0] = make_uint2(w[0], w[1]);
          to[1] = make_uint2(w[2], w[3]);
        }
      }
    __syncthreads();   // vs is used again
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
                               cudaStream_t stream, bool beside) {
  if (T <= 0) return cudaSuccess;
  if (!lora_group_ok(g) || ldx % 8 != 0) return cudaErrorInvalidValue;
  int groups = 0;
  for (int m = 0; m < g.n_mods; ++m) groups += g.mod[m].Rm / LORA_RPC;
  return launch_k(lora_shrink_kernel, dim3((T + LORA_ST - 1) / LORA_ST, groups, lora_passes_apart(T)), dim3(256), 0, stream, x, ldx, tok_slot,
                  g, v, T, beside ? 1 : 0);
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
