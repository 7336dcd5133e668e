// Y = X W^T on CTA pairs (tcgen05 cta_group::2): the products of prompts and of expert segments.
//
// Two neighbouring SMs work on one tile of 256 weight rows x up to 256 tokens.  Weights are the MMA's A operand (each CTA
// holds 128 of the 256 rows), tokens its B operand (each CTA holds half of them and the tensor cores read both halves), so a
// k-block costs an SM 16 KB of weights and at most 16 KB of tokens for 128 x 256 x 64 multiply-adds: two thirds of what the
// one-CTA tile of gemm_tcgen05.cu (128 x 256) reads.  That traffic out of L2 (about 10 TB/s) is what bounds a product of
// thousands of tokens; measured on one B200, T x N x K, one-CTA tiles -> pairs:
//   2048 x 28672 x 4096 (SwiGLU) 742 -> 312 us (1540 TFLOP/s)      512 x 28672 x 4096 (SwiGLU) 335 -> 99 us
//   2048 x 4096 x 14336          218 -> 165 us (1460)              512 x 4096 x 14336           75 -> 55 us
//   2048 x 6144 x 4096           142 -> 84 us (1220)               2048 x 2128 x 2048 (fp32 out)  47 -> 17 us
//   2048 x 4096 x 4096            90 -> 48 us (1440)               257 x 768 x 3072              37 -> 13 us
//
// Token tiles have any size that is a multiple of 32 (UMMA_N), which serves two ends:
//  * dense products: the tokens are cut into the number of equal tiles that fills whole waves of the 74 pairs best
//    (gemm_pair_plan); no tile is ever split along k, so there is no reduction between CTAs and an output is one sum in
//    ascending k whatever the launch;
//  * grouped products (one row segment per expert): a segment is cut into equal tiles of at most 256 rows, a segment of 40
//    rows costs 64 columns.  The tile list is derived from the segment offsets on the device.  In a decode step (three rows
//    an expert) the launch streams the experts' weights at HBM rate, with thousands of tokens it is bound like the dense one.
//
// Roles per CTA: warp 0 TMA producer, warp 1 MMA issuer (leader CTA only) and TMEM owner, warps 2..5 epilogue on a double
// buffered accumulator (2 x 256 columns).  The leader's `full` barrier counts both CTAs' bytes; tcgen05.commit releases a
// ring slot in both CTAs at once.  No wait is unbounded: after about two seconds a role gives up, raises the host-visible
// error word and leaves; copies and MMAs that are still in flight land first, and TMEM is freed on every path.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace tgis {
namespace {

constexpr int PAIR_THREADS = 192;
constexpr int PAIR_BK = 64;
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_TILE_BYTES = 128 * PAIR_BK * 2;         // one CTA's half of either operand
constexpr int PAIR_UNIT = 32;                              // token tiles are multiples of this (UMMA_N step of an M = 256 pair)
constexpr int X_BOX_BYTES = GEMM_X_BOX_MANY * PAIR_BK * 2;
constexpr int PAIR_MAX_GROUPS = 2048;
constexpr int PAIR_BAR_BYTES = 256;
constexpr size_t pair_smem(bool grouped) {
  return (size_t)PAIR_STAGES * 2 * PAIR_TILE_BYTES + 1024 + PAIR_BAR_BYTES + (grouped ? (PAIR_MAX_GROUPS + 1) * sizeof(int) : 0);
}

struct PairArgs {
  void* Y;
  int ldy, T, N, K;
  int n_tiles, x_tiles;     // weight tiles of 256 rows; token tiles (dense)
  int y_f32, mode;          // mode: PAIR_* (Y in fp32: PAIR_PLAIN only)
  const int* seg_off;       // grouped: [n_groups + 1]
  int n_groups;
  const float* row_scale;   // PAIR_RELU2: scale of the input row gather[p] (null: 1)
  const int* gather;
  int* err;                 // host-visible error word
  int batch, x_cs;          // dense: problems side by side (0 or 1: one); columns of X between them (W: N rows, Y: y_bs elements)
  long long y_bs;
  int scale_ld;             // PAIR_ROWSCALE: scale of token t and problem z: row_scale[t * scale_ld + z]
  int late;                 // dense: the next kernel starts once X is final
};

// ---------------------------------------------------------------- cta_group::2 forms
template <uint32_t kCols>
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(smem_dst)), "n"(kCols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n");
}
template <uint32_t kCols>
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "n"(kCols));
}
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the barrier at this offset in both CTAs of the pair once all MMAs issued so far have retired
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}
// tile into this CTA's shared memory, bytes counted on a barrier of either CTA of the pair (`bar`: shared::cluster address)
__device__ __forceinline__ void tma_load_pair(const CUtensorMap* m, uint32_t bar, void* dst, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];\n" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > 4000000000ll) {   // about two seconds: no wait of a working pipeline is that long
      *reinterpret_cast<volatile int*>(err) = 1;
      __threadfence_system();
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ float pair_geglu(float g, float u) {
  return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
}
template <int MODE>
__device__ __forceinline__ float pair_act(float v, float s) {
  if constexpr (MODE == PAIR_RELU2) {
    const float z = fmaxf(v * s, 0.f);
    return z * z;
  } else if constexpr (MODE == PAIR_TANH) {
    return tanhf(v);
  } else if constexpr (MODE == PAIR_ROWSCALE) {
    return v * s;
  } else if constexpr (MODE == PAIR_GELU) {
    return 0.5f * v * (1.f + erff(v * 0.7071067811865476f));
  } else {
    return v;
  }
}
template <class OT>
__device__ __forceinline__ OT pair_out(float v) {
  if constexpr (sizeof(OT) == 4) return v;
  else return __float2bfloat16_rn(v);
}

struct PairTile {
  int w_row;       // first weight row of the tile in the weight map
  int n0;          // first output column
  int row0, rows;  // token rows [row0, row0 + rows)
  int n;           // UMMA_N: rows rounded up to PAIR_UNIT
  int z;           // problem
};

// Tiles of one pair in launch order: index pair, pair + pairs, ...
template <bool GROUPED>
struct PairIter {
  const PairArgs& a;
  const int* start;  // grouped: first tile of every segment [n_groups + 1] (shared memory)
  int i, step, total, g;
  __device__ PairIter(const PairArgs& a_, const int* start_, int pair, int pairs) : a(a_), start(start_), i(pair), step(pairs), g(0) {
    total = GROUPED ? start[a.n_groups] : a.n_tiles * a.x_tiles * max(a.batch, 1);
  }
  __device__ bool next(PairTile& t) {
    if (i >= total) return false;
    int n_tile, x_tile, x_tiles, base, rows, units;
    if (GROUPED) {
      while (i >= start[g + 1]) ++g;
      base = a.seg_off[g];
      rows = a.seg_off[g + 1] - base;
      units = (rows + PAIR_UNIT - 1) / PAIR_UNIT;
      x_tiles = (units + 7) / 8;
      const int k = i - start[g];   // token tile fastest: the pairs that share a weight tile run side by side
      n_tile = k / x_tiles;
      x_tile = k - n_tile * x_tiles;
    } else {
      // blocks of 8 weight tiles, token tile next, weight tile fastest: a wave of 74 is a compact rectangle
      constexpr int NB = 8;
      base = 0;
      rows = a.T;
      units = (rows + PAIR_UNIT - 1) / PAIR_UNIT;
      x_tiles = a.x_tiles;
      const int each = a.n_tiles * x_tiles, z = i / each, k = i - z * each;
      const int full = NB * x_tiles, nb = k / full, rem = k - nb * full, nb_n = min(NB, a.n_tiles - nb * NB);
      t.z = z;
      x_tile = rem / nb_n;
      n_tile = nb * NB + rem - x_tile * nb_n;
    }
    const int u0 = x_tile * units / x_tiles, u1 = (x_tile + 1) * units / x_tiles;
    t.n0 = n_tile * 256;
    if (GROUPED) t.z = 0;
    t.w_row = (GROUPED ? g : t.z) * a.N + t.n0;
    t.row0 = base + u0 * PAIR_UNIT;
    t.rows = min(rows - u0 * PAIR_UNIT, (u1 - u0) * PAIR_UNIT);
    t.n = (u1 - u0) * PAIR_UNIT;
    i += step;
    return true;
  }
};

// One accumulator (this warp's 32 weight rows x t.rows tokens) -> Y; lane = weight row, column = token
template <int MODE, class OT>
__device__ __forceinline__ void pair_store(const PairArgs& a, const PairTile& t, int n, uint32_t taddr, int lane) {
  constexpr bool GLU = MODE == PAIR_SWIGLU || MODE == PAIR_SWIGLU_BF16 || MODE == PAIR_GEGLU;
  const bool n_ok = GLU ? (n | 1) < a.N : n < a.N;
  OT* y = reinterpret_cast<OT*>(a.Y) + (size_t)t.z * a.y_bs + (size_t)t.row0 * a.ldy + (GLU ? n >> 1 : n);
#pragma unroll 1
  for (int c0 = 0; c0 < t.rows; c0 += 32, y += (size_t)32 * a.ldy) {
    uint32_t r[32];
    // the scale of token c0 + lane: one load in flight for 32 tokens, not one behind the other per token (4096 rows of 1024 x 2048 in 8
    // segments 77 -> 22 us; 16 heads of 128 x 512 at 2048 tokens 97 -> 18)
    float scale = 1.f;
    if constexpr (MODE == PAIR_RELU2) {
      if (a.row_scale != nullptr && c0 + lane < t.rows) scale = a.row_scale[a.gather != nullptr ? a.gather[t.row0 + c0 + lane] : t.row0 + c0 + lane];
    } else if constexpr (MODE == PAIR_ROWSCALE) {
      if (c0 + lane < t.rows) scale = a.row_scale[(size_t)(t.row0 + c0 + lane) * a.scale_ld + t.z];
    }
    tmem_ld_32x32b_x16(taddr + c0, r);
    tmem_ld_32x32b_x16(taddr + c0 + 16, r + 16);
    tmem_ld_wait();
    const int valid = n_ok ? t.rows - c0 : 0;
    if constexpr (GLU) {
      // rows (2j, 2j + 1) of W are (gate_j, up_j), in adjacent lanes: the even lane makes token c's value, the odd lane token
      // c + 1's, with one exchange for both
      const bool odd = lane & 1;
      OT* yl = y + (odd ? a.ldy : 0);
      const int mine_valid = valid - (odd ? 1 : 0);
      float g[16], u[16], v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? r[2 * j] : r[2 * j + 1]), 1);
        g[j] = odd ? got : __uint_as_float(r[2 * j]);
        u[j] = odd ? __uint_as_float(r[2 * j + 1]) : got;
        if (!n_ok) g[j] = 0.f;   // (whatever such a row holds does not send the warp into a division)
      }
      if constexpr (MODE == PAIR_SWIGLU_BF16) {   // the rounding points of a bf16 gate / up product followed by silu and a product
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = bf16_round(g[j]);
        silu_bf16_n(g, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] *= bf16_round(u[j]);
      } else if constexpr (MODE == PAIR_SWIGLU) {
        silu_mul_bf16_n(g, u, v, mine_valid <= 0 ? 0u : 0xffffu >> (16 - min((mine_valid + 1) / 2, 16)));   // tokens 2 j < mine_valid
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = pair_geglu(g[j], u[j]);
      }
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (2 * j < mine_valid) yl[(size_t)(2 * j) * a.ldy] = pair_out<OT>(v[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        float s = 1.f;
        if constexpr (MODE == PAIR_RELU2 || MODE == PAIR_ROWSCALE) s = __shfl_sync(0xffffffffu, scale, j);
        if (j < valid) y[(size_t)j * a.ldy] = pair_out<OT>(pair_act<MODE>(__uint_as_float(r[j]), s));
      }
    }
  }
}

template <bool GROUPED>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ PairArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_w = smem;
  uint8_t* smem_x = smem + PAIR_STAGES * PAIR_TILE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + 2 * PAIR_STAGES * PAIR_TILE_BYTES);
  uint64_t* empty_bar = full_bar + PAIR_STAGES;
  uint64_t* tmem_full = empty_bar + PAIR_STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_base_smem + 1);   // some role's wait ran out
  int* seg_start = reinterpret_cast<int*>(smem + 2 * PAIR_STAGES * PAIR_TILE_BYTES + PAIR_BAR_BYTES);

  const int warp = threadIdx.x >> 5, lane = (int)lane_id();
  const int rank = (int)cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int KB = (a.K + PAIR_BK - 1) / PAIR_BK;

  if (warp == 0 && elect_one()) {
    tma_prefetch_desc(&wmap);
    tma_prefetch_desc(&xmap);
  }
  if (warp == 1) {
    if (elect_one()) {
      for (int i = 0; i < PAIR_STAGES; ++i) {
        mbar_init(&full_bar[i], 1);    // the leader's expect_tx (both CTAs' bytes)
        mbar_init(&empty_bar[i], 1);   // commit_pair
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&tmem_full[i], 1);   // commit_pair
        mbar_init(&tmem_empty[i], 8);  // four epilogue warps of either CTA (leader's barrier)
      }
      *gave_up = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc_pair<512>(tmem_base_smem);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_smem;
  if (!a.late) griddep_launch();
  if (GROUPED) {   // the segment offsets come from a kernel of this step
    griddep_wait();
    if (warp == 0) {   // exclusive prefix sum of the segments' tile counts
      int run = 0;
      for (int g0 = 0; g0 < a.n_groups; g0 += 32) {
        const int g = g0 + lane;
        int c = 0;
        if (g < a.n_groups) c = ((a.seg_off[g + 1] - a.seg_off[g] + PAIR_UNIT - 1) / PAIR_UNIT + 7) / 8 * a.n_tiles;
        int s = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, s, o);
          if (lane >= o) s += up;
        }
        if (g < a.n_groups) seg_start[g] = run + s - c;
        run += __shfl_sync(0xffffffffu, s, 31);
      }
      if (lane == 0) seg_start[a.n_groups] = run;
    }
    __syncthreads();
  }

  if (warp == 0) {
    // ===================== TMA producer (both CTAs) =====================
    if (elect_one()) {
      PairIter<GROUPED> it(a, seg_start, pair, pairs);
      PairTile t;
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t full0 = dsmem_addr(smem_u32(full_bar), 0);   // the leader's barriers
      int w_row = 0, x_row = 0, x_col = 0, boxes = 0;
      uint32_t bytes = 0;
      auto set_tile = [&]() {
        boxes = (t.n / 2 + GEMM_X_BOX_MANY - 1) / GEMM_X_BOX_MANY;
        bytes = 2u * (uint32_t)(PAIR_TILE_BYTES + boxes * X_BOX_BYTES);
        w_row = t.w_row + rank * 128;
        x_row = t.row0 + rank * (t.n / 2);
        x_col = t.z * a.x_cs;
      };
      auto load_w = [&](int s, int kb) {
        if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], bytes);
        tma_load_pair(&wmap, full0 + s * 8, smem_w + s * PAIR_TILE_BYTES, kb * PAIR_BK, w_row);
      };
      auto load_x = [&](int s, int kb) {
#pragma unroll
        for (int b = 0; b < 128 / GEMM_X_BOX_MANY; ++b)
          if (b < boxes) tma_load_pair(&xmap, full0 + s * 8, smem_x + s * PAIR_TILE_BYTES + b * X_BOX_BYTES, x_col + kb * PAIR_BK, x_row + b * GEMM_X_BOX_MANY);
      };
      bool have = it.next(t);
      if (have) set_tile();
      if (!GROUPED) {
        // weights are static: the first ring of them is requested before the previous kernel has finished
        const int pre = have ? min(KB, PAIR_STAGES) : 0;
        for (int kb = 0; kb < pre; ++kb) load_w(kb, kb);
        griddep_wait();
        if (a.late) griddep_launch_after();
        for (int kb = 0; kb < pre; ++kb) load_x(kb, kb);
        issued = pre;
        stage = pre % PAIR_STAGES;
        phase = pre == PAIR_STAGES ? 1 : 0;
      }
      while (have && ok) {
        for (int kb = issued; kb < KB; ++kb) {
          if (!(ok = pair_wait(&empty_bar[stage], phase ^ 1, a.err))) break;
          load_w(stage, kb);
          load_x(stage, kb);
          if (++stage == PAIR_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        issued = 0;
        have = it.next(t);
        if (have) set_tile();
      }
      if (!ok) *gave_up = 1;
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (leader) =====================
    if (rank == 0 && elect_one()) {
      PairIter<GROUPED> it(a, seg_start, pair, pairs);
      PairTile t;
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      while (ok && it.next(t)) {   // (one thread: 257 tokens x 4096 x 14336 56.3 us with a warp's votes at every k-block, 54.1 without)
        const uint32_t idesc = make_idesc_bf16(256, (uint32_t)t.n);
        if (!(ok = pair_wait(&tmem_empty[acc], acc_phase ^ 1, a.err))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int kb = 0; kb < KB; ++kb) {
          if (!(ok = pair_wait(&full_bar[stage], phase, a.err))) break;
          tc_fence_after();
          const uint64_t a_desc = make_smem_desc_sw128(smem_u32(smem_w + stage * PAIR_TILE_BYTES));
          const uint64_t b_desc = make_smem_desc_sw128(smem_u32(smem_x + stage * PAIR_TILE_BYTES));
#pragma unroll
          for (int k = 0; k < PAIR_BK / 16; ++k)
            mma_pair(d_tmem, a_desc + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          commit_pair(&empty_bar[stage]);
          if (++stage == PAIR_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) commit_pair(&tmem_full[acc]);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
      if (!ok) *gave_up = 1;
    }
  } else {
    // ===================== epilogue (both CTAs): lane = weight row, column = token =====================
    const int sub = warp & 3;
    PairIter<GROUPED> it(a, seg_start, pair, pairs);
    PairTile t;
    int acc = 0;
    uint32_t acc_phase = 0;
    if (!GROUPED) griddep_wait();   // Y (and the input scales) may still be in use by the previous kernels
    while (it.next(t)) {
      if (!__all_sync(0xffffffffu, pair_wait(&tmem_full[acc], acc_phase, a.err))) {
        if (lane == 0) *gave_up = 1;
        break;
      }
      tc_fence_after();
      const int n = t.n0 + rank * 128 + sub * 32 + lane;
      const uint32_t taddr = tmem_base + acc * 256 + ((uint32_t)(sub * 32) << 16);
      using bf = __nv_bfloat16;
      switch (a.mode) {
        case PAIR_SWIGLU_BF16: pair_store<PAIR_SWIGLU_BF16, bf>(a, t, n, taddr, lane); break;
        case PAIR_SWIGLU: pair_store<PAIR_SWIGLU, bf>(a, t, n, taddr, lane); break;
        case PAIR_GEGLU: pair_store<PAIR_GEGLU, bf>(a, t, n, taddr, lane); break;
        case PAIR_RELU2: pair_store<PAIR_RELU2, bf>(a, t, n, taddr, lane); break;
        case PAIR_GELU: pair_store<PAIR_GELU, bf>(a, t, n, taddr, lane); break;
        case PAIR_TANH: pair_store<PAIR_TANH, bf>(a, t, n, taddr, lane); break;
        case PAIR_ROWSCALE: pair_store<PAIR_ROWSCALE, bf>(a, t, n, taddr, lane); break;
        default:
          if (a.y_f32) pair_store<PAIR_PLAIN, float>(a, t, n, taddr, lane);
          else pair_store<PAIR_PLAIN, bf>(a, t, n, taddr, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(dsmem_addr(smem_u32(&tmem_empty[acc]), 0));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  // A wait that ran out in any role leaves copies and MMAs of the others behind, all issued by now and done long before this
  // millisecond is over: neither shared memory nor TMEM is given back while they may still write there.  (Where the leader's MMAs
  // stop, the other CTA's epilogue gets no accumulator and comes here too.)
  if (*gave_up)
    for (const long long t0 = clock64(); clock64() - t0 < 2000000ll;) {}
  cluster_sync_all();   // nobody leaves while the peer may still read its shared memory or signal its barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair<512>(tmem_base);
  }
}

// ---------------------------------------------------------------- few tokens: equal shares of weight rows
// A product of up to 256 tokens is bound by its weight bytes, so what counts is that every SM streams the same number of them from
// the first microsecond to the last.  Here a pair's tile has as many rows as make the tiles fill whole waves of pairs (2 R, R even,
// up to 128 a CTA): a CTA loads exactly its R rows, the MMA's other rows read what happens to lie behind them in shared memory and
// go nowhere.  No tile is split along k, so nothing is reduced between CTAs and an output is one sum in ascending k.  Each
// CTA loads half of the tokens, R + n / 2 rows a k-block; gemm_rows_takes says where that is less than what a split along k costs.
// One thread issues all MMAs and a barrier covers two k-blocks: with few tokens a k-block takes no longer than a warp's votes and a
// commit (28672 x 4096 in bf16, 96 tokens, 46 us; 10256 x 2048 15.4 us with a k-block to a barrier, 12.9 with two).  What bounds it
// now: 22528 x 2048 streams its weights at 4.9 TB/s of a launch's 19 us, of which 4 are its start and its end; shares of fewer
// than some 56 rows wait for the 0.16 us that a k-block's MMAs take.
constexpr int ROWS_MAX_STAGES = 24;
constexpr int ROWS_RING = 200 * 1024;
constexpr int ROWS_BAR_BYTES = 512;
constexpr int ROWS_SMEM = ROWS_RING + PAIR_TILE_BYTES + 1024 + ROWS_BAR_BYTES;   // (the last stage's MMA reads 128 rows as well)
struct RowsArgs {
  PairArgs p;
  int R, n, tiles;                  // weight rows of a CTA's share of a tile, UMMA_N, tiles
  int stages, ksub, w_bytes, x_bytes;   // ring; k-blocks of a stage; bytes of one k-block's operands in it (whole 8-row groups)
};
__device__ __forceinline__ void tma_load_pair_hint(const CUtensorMap* m, uint32_t bar, void* dst, int c0, int c1, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;\n" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}

__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ RowsArgs ra) {
  extern __shared__ uint8_t smem_raw[];
  const PairArgs& a = ra.p;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + ROWS_RING + PAIR_TILE_BYTES);
  uint64_t* empty_bar = full_bar + ROWS_MAX_STAGES;
  uint64_t* tmem_full = empty_bar + ROWS_MAX_STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_base_smem + 1);

  const int warp = threadIdx.x >> 5, lane = (int)lane_id();
  const int rank = (int)cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int sub_bytes = ra.w_bytes + ra.x_bytes, stage_bytes = ra.ksub * sub_bytes, KS = a.K / (PAIR_BK * ra.ksub);

  if (warp == 0 && elect_one()) {
    tma_prefetch_desc(&wmap);
    tma_prefetch_desc(&xmap);
  }
  if (warp == 1) {
    if (elect_one()) {
      for (int i = 0; i < ra.stages; ++i) {
        mbar_init(&full_bar[i], 1);
        mbar_init(&empty_bar[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&tmem_full[i], 1);
        mbar_init(&tmem_empty[i], 8);
      }
      *gave_up = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc_pair<512>(tmem_base_smem);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_smem;
  if (!a.late) griddep_launch();

  if (warp == 0) {
    // ===================== TMA producer (both CTAs) =====================
    if (elect_one()) {
      const uint32_t full0 = dsmem_addr(smem_u32(full_bar), 0);   // the leader's barriers
      const uint32_t bytes = 2u * (uint32_t)(ra.ksub * (ra.R + ra.n / 2) * PAIR_BK * 2);
      const uint64_t once = policy_evict_first();
      const int x_row = rank * (ra.n / 2);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      auto load_w = [&](int s, int ks, int w_row) {
        if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], bytes);
        for (int j = 0; j < ra.ksub; ++j)
          tma_load_pair_hint(&wmap, full0 + s * 8, smem + s * stage_bytes + j * sub_bytes, (ks * ra.ksub + j) * PAIR_BK, w_row, once);
      };
      auto load_x = [&](int s, int ks) {
        for (int j = 0; j < ra.ksub; ++j)
          tma_load_pair(&xmap, full0 + s * 8, smem + s * stage_bytes + j * sub_bytes + ra.w_bytes, (ks * ra.ksub + j) * PAIR_BK, x_row);
      };
      // weights are static: the first ring of them is requested before the previous kernel has finished
      const int pre = pair < ra.tiles ? min(KS, ra.stages) : 0;
      for (int ks = 0; ks < pre; ++ks) load_w(ks, ks, (pair * 2 + rank) * ra.R);
      griddep_wait();
      if (a.late) griddep_launch_after();
      for (int ks = 0; ks < pre; ++ks) load_x(ks, ks);
      stage = pre % ra.stages;
      phase = pre == ra.stages ? 1 : 0;
      for (int t = pair, first = pre; t < ra.tiles && ok; t += pairs, first = 0) {
        const int w_row = (t * 2 + rank) * ra.R;
        for (int ks = first; ks < KS; ++ks) {
          if (!(ok = pair_wait(&empty_bar[stage], phase ^ 1, a.err))) break;
          load_w(stage, ks, w_row);
          load_x(stage, ks);
          if (++stage == ra.stages) stage = 0, phase ^= 1;
        }
      }
      if (!ok) *gave_up = 1;
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (leader) =====================
    if (rank == 0 && elect_one()) {   // (one thread from end to end: with few tokens a stage takes no longer than a warp's votes)
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      const uint32_t idesc = make_idesc_bf16(256, (uint32_t)ra.n), ring = smem_u32(smem);
      for (int t = pair; t < ra.tiles && ok; t += pairs) {
        if (!(ok = pair_wait(&tmem_empty[acc], acc_phase ^ 1, a.err))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int ks = 0; ks < KS; ++ks) {
          if (!(ok = pair_wait(&full_bar[stage], phase, a.err))) break;
          tc_fence_after();
          for (int j = 0; j < ra.ksub; ++j) {
            const uint32_t at = ring + stage * stage_bytes + j * sub_bytes;
            const uint64_t a_desc = make_smem_desc_sw128(at), b_desc = make_smem_desc_sw128(at + ra.w_bytes);
#pragma unroll
            for (int k = 0; k < PAIR_BK / 16; ++k)
              mma_pair(d_tmem, a_desc + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (ks > 0 || j > 0 || k > 0) ? 1u : 0u);
          }
          commit_pair(&empty_bar[stage]);
          if (++stage == ra.stages) stage = 0, phase ^= 1;
        }
        if (ok) commit_pair(&tmem_full[acc]);
        if (++acc == 2) acc = 0, acc_phase ^= 1;
      }
      if (!ok) *gave_up = 1;
    }
  } else {
    // ===================== epilogue (both CTAs): lane = weight row, column = token =====================
    const int sub = warp & 3, row = sub * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    griddep_wait();   // Y may still be in use by the previous kernels
    for (int t = pair; t < ra.tiles; t += pairs) {
      if (!__all_sync(0xffffffffu, pair_wait(&tmem_full[acc], acc_phase, a.err))) {
        if (lane == 0) *gave_up = 1;
        break;
      }
      tc_fence_after();
      if (sub * 32 < ra.R) {
        PairTile pt;
        pt.n0 = 0; pt.w_row = 0; pt.z = 0;
        pt.row0 = 0; pt.rows = a.T; pt.n = ra.n;
        const int n = row < ra.R ? (t * 2 + rank) * ra.R + row : a.N;
        const uint32_t taddr = tmem_base + acc * 256 + ((uint32_t)(sub * 32) << 16);
        using bf = __nv_bfloat16;
        switch (a.mode) {
          case PAIR_SWIGLU_BF16: pair_store<PAIR_SWIGLU_BF16, bf>(a, pt, n, taddr, lane); break;
          case PAIR_GEGLU: pair_store<PAIR_GEGLU, bf>(a, pt, n, taddr, lane); break;
          case PAIR_RELU2: pair_store<PAIR_RELU2, bf>(a, pt, n, taddr, lane); break;
          default:
            if (a.y_f32) pair_store<PAIR_PLAIN, float>(a, pt, n, taddr, lane);
            else pair_store<PAIR_PLAIN, bf>(a, pt, n, taddr, lane);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(dsmem_addr(smem_u32(&tmem_empty[acc]), 0));
      if (++acc == 2) acc = 0, acc_phase ^= 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*gave_up)   // as in gemm_pair_kernel
    for (const long long t0 = clock64(); clock64() - t0 < 2000000ll;) {}
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair<512>(tmem_base);
  }
}

// host-visible error word, one for the process (a raised word is an error of the process's device, as a sticky CUDA error is).
// Pinned memory cannot be had while a stream is being captured, so an engine has it made before its first step
// (gemm_pair_prepare); a refusal is not remembered.
std::atomic<int*> pair_word{nullptr};
cudaError_t make_pair_word() {
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  if (pair_word.load(std::memory_order_acquire) != nullptr) return cudaSuccess;
  int* p = nullptr;
  const cudaError_t e = cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
  if (e != cudaSuccess) return e;
  *p = 0;
  pair_word.store(p, std::memory_order_release);
  return cudaSuccess;
}

std::atomic<int> pair_launches{0}, pair_fault_in{0};   // gemm_pair_fault

// the error word for one launch (and the host's stand-in for a wait of it that runs out, gemm_pair_fault)
cudaError_t claim_pair_word(int*& err) {
  const cudaError_t word = gemm_pair_prepare();
  if (word != cudaSuccess) return word;
  err = pair_word.load(std::memory_order_acquire);
  pair_launches.fetch_add(1, std::memory_order_relaxed);
  if (pair_fault_in.load(std::memory_order_relaxed) > 0 && pair_fault_in.fetch_sub(1) == 1) *reinterpret_cast<volatile int*>(err) = 1;
  return cudaSuccess;
}

template <bool GROUPED>
cudaError_t launch_pair(const CUtensorMap& wmap, const CUtensorMap& xmap, PairArgs a, int grid, cudaStream_t stream) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(gemm_pair_kernel<GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pair_smem(GROUPED));
  if (attr != cudaSuccess) return attr;
  const cudaError_t word = claim_pair_word(a.err);
  if (word != cudaSuccess) return word;
  return launch_k_cluster(gemm_pair_kernel<GROUPED>, dim3(grid), dim3(PAIR_THREADS), pair_smem(GROUPED), stream, 2, wmap, xmap, a);
}

}  // namespace

cudaError_t gemm_pair_prepare() { return pair_word.load(std::memory_order_acquire) != nullptr ? cudaSuccess : make_pair_word(); }

cudaError_t gemm_pair_word(int** word) {
  const cudaError_t e = gemm_pair_prepare();
  *word = pair_word.load(std::memory_order_acquire);
  return e;
}

bool gemm_pair_failed() {
  const int* w = pair_word.load(std::memory_order_acquire);
  return w != nullptr && *reinterpret_cast<const volatile int*>(w) != 0;
}

int gemm_pair_fault(int nth) {
  if (int* w = pair_word.load(std::memory_order_acquire)) *reinterpret_cast<volatile int*>(w) = 0;
  pair_fault_in.store(nth);
  return pair_launches.exchange(0);
}

// Number of token tiles for a dense product of T tokens and N weight rows on `pairs` CTA pairs.  A k-block of a tile of n
// tokens takes about 130 + n nanoseconds when all pairs run (2048 x 28672 x 4096: 382 at n = 256, 339 at 224, 284 at 192,
// 245 at 128; below 64 the weight half alone is what it takes), so the count that makes waves * (130 + largest n) smallest
// is taken.  Measured at the sizes of an 8B layer and of 768 to 2048 wide ones, 257 to 2048 tokens: within 3 % of the best
// count but for 2048 x 6144 x 4096 (8 tiles 84 us, 11 tiles 74 us).
int gemm_pair_plan(int T, int N, int pairs) {
  const int units = (T + PAIR_UNIT - 1) / PAIR_UNIT, n_tiles = (N + 255) / 256, least = (units + 7) / 8;
  int best = least;
  long long best_cost = -1;
  for (int x = least; x <= units && x <= least + 16; ++x) {
    const int n = (units + x - 1) / x * PAIR_UNIT;
    const long long cost = ((long long)n_tiles * x + pairs - 1) / pairs * (130 + (n > 64 ? n : 64));
    if (best_cost < 0 || cost < best_cost) {
      best = x;
      best_cost = cost;
    }
  }
  return best;
}

cudaError_t gemm_pair_launch(const CUtensorMap& wmap, const CUtensorMap& xmap, void* Y, int ldy, int y_f32, int mode, int T, int N, int K,
                             int num_sms, cudaStream_t stream, bool late) {
  if (T <= 0 || N <= 0 || K <= 0 || (y_f32 && mode != PAIR_PLAIN)) return cudaErrorInvalidValue;
  const int pairs = num_sms / 2;
  if (pairs < 1) return cudaErrorInvalidValue;
  PairArgs a{};
  a.Y = Y; a.ldy = ldy; a.T = T; a.N = N; a.K = K;
  a.y_f32 = y_f32; a.mode = mode; a.late = late;
  a.n_tiles = (N + 255) / 256;
  a.x_tiles = gemm_pair_plan(T, N, pairs);
  const int tiles = a.n_tiles * a.x_tiles;
  return launch_pair<false>(wmap, xmap, a, 2 * (tiles < pairs ? tiles : pairs), stream);
}

// Dense products of prompts that gemm_bf16_launch's layout does not cover: one per head side by side in the columns of X, few weight
// rows (a router), a tanh, a scale per row and problem.  mma.sync tiles -> here, microseconds at 300 and 2048 tokens: 16 heads of
// 512 x 128 14.0 -> 6.7 and 55 -> 20, 16 of 128 x 512 with scales 19.6 -> 7.7 and 28 -> 18, 65 x 2048 48 -> 10 and 48 -> 11, tanh 64 x 2048
// 53 -> 13 and 53 -> 15, 2048 x 64 11.6 -> 5.2 and 12.9 -> 7.4; the errors against 64 bits are equal to all digits.  Up to 256 tokens the
// register products and the warp per output have them; fewer than 32 weight rows would fill an eighth of a tile.
bool gemm_pair_takes_dense(const GemmAny& a) {
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const int batch = a.batch > 1 ? a.batch : 1;
  const bool mode_ok = a.mode == GEMM_ANY_PLAIN || (a.y_dtype == DT_BF16 && (a.mode == GEMM_ANY_TANH || a.mode == GEMM_ANY_ROWSCALE));
  return mode_ok && a.seg_off == nullptr && a.gather == nullptr && a.T > 256 && a.N >= 32 && a.K >= PAIR_BK && a.K % PAIR_BK == 0 &&
         a.x_dtype == DT_BF16 && a.w_dtype == DT_BF16 && a.ldw == a.K && a.ldx % 8 == 0 && a.ldx >= a.K && al16(a.X) && al16(a.W) &&
         (batch == 1 || (a.w_bs == (long long)a.N * a.K && a.x_bs % 8 == 0 && a.x_bs >= 0 && (long long)(batch - 1) * a.x_bs + a.K <= a.ldx)) &&
         (long long)batch * a.N < (1ll << 31);
}
cudaError_t gemm_pair_dense_launch(const GemmAny& g, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int batch = g.batch > 1 ? g.batch : 1, pairs = sms / 2;
  if (pairs < 1) return cudaErrorInvalidValue;
  const uint64_t cols = (uint64_t)g.K + (batch > 1 ? (uint64_t)(batch - 1) * g.x_bs : 0);
  CUtensorMap wm, xm;
  if (make_tmap_bf16_2d(&wm, g.W, (uint64_t)batch * g.N, g.K, g.K, 128, PAIR_BK) != 0 ||
      make_tmap_bf16_2d(&xm, g.X, g.T, cols, g.ldx, GEMM_X_BOX_MANY, PAIR_BK) != 0)
    return cudaErrorInvalidValue;
  PairArgs a{};
  a.Y = g.Y; a.ldy = g.ldy; a.T = g.T; a.N = g.N; a.K = g.K;
  a.y_f32 = g.y_dtype == DT_F32;
  a.mode = g.mode == GEMM_ANY_TANH ? PAIR_TANH : g.mode == GEMM_ANY_ROWSCALE ? PAIR_ROWSCALE : PAIR_PLAIN;
  a.n_tiles = (g.N + 255) / 256;
  a.x_tiles = gemm_pair_plan(g.T, a.n_tiles * 256 * batch, pairs);
  a.row_scale = g.row_scale; a.scale_ld = g.scale_ld;
  a.batch = batch; a.x_cs = batch > 1 ? (int)g.x_bs : 0; a.y_bs = batch > 1 ? g.y_bs : 0;
  const long long tiles = (long long)a.n_tiles * a.x_tiles * batch;
  return launch_pair<false>(wm, xm, a, 2 * (int)(tiles < pairs ? tiles : pairs), stream);
}

// The share of a product of N weight rows that one CTA of a pair takes: whole waves of pairs, an even number of rows
static int rows_share(int N, int pairs) {
  const int waves = (N + 256 * pairs - 1) / (256 * pairs), per = (N + 2 * pairs * waves - 1) / (2 * pairs * waves);
  return (per + 1) & ~1;
}
// At least 40 rows a CTA up to 64 tokens, four from there (fewer rows: the cut along k or the pairs' token tiles are ahead); beyond 128
// tokens only where the rows fill more than one wave; a long k only where its bytes take longer than its MMAs.  The measured
// table stands at gemm_takes_pairs.  Every line in T is one at which the token tiles change anyway: a row's bits change nowhere else.
bool gemm_rows_takes(int T, int N, int K, int num_sms) {
  if (T <= 16 || T > 256 || K % PAIR_BK != 0 || num_sms < 2) return false;
  const int pairs = num_sms / 2, R = rows_share(N, pairs);
  if (R < 56 && K > 4096) return false;
  // (In a chain of kernels the cut along k is ahead up to 32 tokens: its ring is under way sooner.  Eight 8B layers, 24 decode steps, ms, cut
  // -> shares, at 33, 40 and 48 requests: 34.6 -> 33.7, 36.7 -> 35.8, 39.3 -> 38.3; at 56 and 64 without shares 42.1 and 45.6, with 40.4 and 43.7.)
  if (T <= 32 && K > 2048) return false;
  return T <= 128 ? R >= 40 || (T > 64 && N >= 8 * pairs) : N > 256 * pairs;
}
cudaError_t gemm_rows_launch(const void* X, const void* W, void* Y, int ldy, int y_f32, int mode, int T, int N, int K, int num_sms,
                             cudaStream_t stream, bool late) {
  if (!gemm_rows_takes(T, N, K, num_sms) || (y_f32 && mode != PAIR_PLAIN)) return cudaErrorInvalidValue;
  const int pairs = num_sms / 2;
  RowsArgs ra{};
  PairArgs& a = ra.p;
  a.Y = Y; a.ldy = ldy; a.T = T; a.N = N; a.K = K;
  a.y_f32 = y_f32; a.mode = mode; a.late = late;
  ra.R = rows_share(N, pairs);
  ra.n = (T + PAIR_UNIT - 1) / PAIR_UNIT * PAIR_UNIT;
  ra.tiles = (N + 2 * ra.R - 1) / (2 * ra.R);
  ra.w_bytes = (ra.R + 7) / 8 * 1024;
  ra.x_bytes = ra.n / 2 * PAIR_BK * 2;
  ra.ksub = K % (2 * PAIR_BK) == 0 ? 2 : 1;   // (a barrier costs the issuing thread as much as two k-blocks of few tokens)
  ra.stages = std::min(ROWS_RING / (ra.ksub * (ra.w_bytes + ra.x_bytes)), ROWS_MAX_STAGES);
  CUtensorMap wm, xm;
  if (make_tmap_bf16_2d(&wm, W, N, K, K, ra.R, PAIR_BK) != 0 || make_tmap_bf16_2d(&xm, X, T, K, K, ra.n / 2, PAIR_BK) != 0)
    return cudaErrorInvalidValue;
  static const cudaError_t attr = cudaFuncSetAttribute(gemm_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM);
  if (attr != cudaSuccess) return attr;
  const cudaError_t word = claim_pair_word(a.err);
  if (word != cudaSuccess) return word;
  return launch_k_cluster(gemm_rows_kernel, dim3(2 * std::min(ra.tiles, pairs)), dim3(PAIR_THREADS), ROWS_SMEM, stream, 2, wm, xm, ra);
}

// X rows of a grouped product in segment order: out[p] = X[gather[p] / div], p < seg_off[n_groups]
__global__ void __launch_bounds__(256) gather_segment_rows_kernel(const uint4* __restrict__ X, int ldx16, const int* __restrict__ gather, int div,
                                                                  const int* __restrict__ seg_end, uint4* __restrict__ out, int row16) {
  griddep_launch();
  griddep_wait();
  const int p = blockIdx.x;
  if (p >= *seg_end) return;
  const uint4* src = X + (size_t)(gather[p] / div) * ldx16;
  uint4* dst = out + (size_t)p * row16;
  for (int c = threadIdx.x; c < row16; c += 256) dst[c] = src[c];
}

// Whether a grouped product runs here.  The operands' rows start on 16-byte boundaries and the segments' weight matrices lie
// one behind the other (one tensor map covers them); gathered rows need room to be laid out in segment order first
// (12288 rows x 2048: 16 us against 660 us for the product that read them one by one).
bool gemm_pair_takes_groups(const GemmAny& a) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const bool mode_ok = a.mode == GEMM_ANY_PLAIN || (a.y_dtype == DT_BF16 && (a.mode == GEMM_ANY_SWIGLU || a.mode == GEMM_ANY_GEGLU ||
                                                                            a.mode == GEMM_ANY_RELU2 || a.mode == GEMM_ANY_GELU));
  return mode_ok && a.seg_off != nullptr && a.batch <= 1 && a.x_dtype == DT_BF16 && a.w_dtype == DT_BF16 && a.n_groups >= 1 &&
         a.n_groups <= PAIR_MAX_GROUPS && a.w_gs == (long long)a.N * a.ldw && (long long)a.n_groups * a.N < (1ll << 31) && a.K >= PAIR_BK &&
         a.K % 8 == 0 && a.ldx % 8 == 0 && a.ldw % 8 == 0 && a.ldx >= a.K && a.ldw >= a.K && al16(a.X) && al16(a.W) &&
         (a.gather == nullptr || (a.gather_div > 0 && al16(a.gather_ws) && a.gather_ws != nullptr && a.gather_ws_bytes >= (size_t)a.T * a.K * 2));
}

cudaError_t gemm_pair_grouped_launch(const GemmAny& g, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const void* X = g.X;
  int ldx = g.ldx;
  if (g.gather != nullptr) {
    e = launch_k(gather_segment_rows_kernel, dim3(g.T), dim3(256), 0, stream, (const uint4*)g.X, g.ldx / 8, g.gather, g.gather_div,
                 g.seg_off + g.n_groups, (uint4*)g.gather_ws, g.K / 8);
    if (e != cudaSuccess) return e;
    X = g.gather_ws;
    ldx = g.K;
  }
  CUtensorMap wm, xm;
  if (make_tmap_bf16_2d(&wm, g.W, (uint64_t)g.n_groups * g.N, g.K, g.ldw, 128, PAIR_BK) != 0 ||
      make_tmap_bf16_2d(&xm, X, g.T, g.K, ldx, GEMM_X_BOX_MANY, PAIR_BK) != 0)
    return cudaErrorInvalidValue;
  PairArgs a{};
  a.Y = g.Y; a.ldy = g.ldy; a.T = g.T; a.N = g.N; a.K = g.K;
  a.y_f32 = g.y_dtype == DT_F32;
  a.mode = g.mode == GEMM_ANY_SWIGLU ? PAIR_SWIGLU : g.mode == GEMM_ANY_GEGLU ? PAIR_GEGLU : g.mode == GEMM_ANY_RELU2 ? PAIR_RELU2
           : g.mode == GEMM_ANY_GELU ? PAIR_GELU : PAIR_PLAIN;
  a.n_tiles = (g.N + 255) / 256;
  a.seg_off = g.seg_off; a.n_groups = g.n_groups;
  a.row_scale = g.row_scale; a.gather = g.gather;
  const int pairs = sms / 2;
  // at most one tile per started 256 rows of every segment: fewer tiles than pairs leave the rest without work
  const long long most = (long long)a.n_tiles * (g.T / 256 + (g.n_groups < g.T ? g.n_groups : g.T));
  return launch_pair<true>(wm, xm, a, 2 * (int)(most < pairs ? (most < 1 ? 1 : most) : pairs), stream);
}

}  // namespace tgis
