// Latent attention of prompts in head space, on tcgen05 (LatentGeom with 128 + 64 query and 128 value dims a head, bf16).
//
// attention_latent.cu folds the up-projections of keys and values into query and output, so that all heads of a token read one cached
// row: right for single tokens, which are bound by those rows.  A prompt's tokens share keys, and there the folded form multiplies
// 576 + 512 numbers for a (query, key, head) where the heads' own keys and values have 192 + 128, on top of a folded query of fp32 [T, heads,
// 576].  Here a portion's keys and values are made once (latent_rows_launch gathers the cached rows, one product makes the heads' plain
// keys and values from them; the rotary part is the cached one, for all heads) and then attended to like any other:
//
// A unit of work is 256 query tokens of one sequence and head; 128 of them fill one M = 128 accumulator, and both accumulators of the CTA
// read every K and V tile of 128 keys that was staged once.  One CTA per SM walks the units, longest first in snake order.  S = Q K^T
// goes to TMEM; a thread per row takes its 128 scores and leaves bf16 probabilities in their place, which the tensor cores read from
// there: O += P V.  The two accumulators alternate, so one's softmax runs under the other's products.  The running maximum that a row's sums
// refer to moves only when a score exceeds it by 2^8, and only then O is scaled (the conditional rescaling published with
// FlashAttention-4).  Tiles are counted from the sequence's first token: a row's bits do not depend on its company.  A row that
// comes out with numbers that are not finite although no key that it sees has them (the tensor cores add 0 * V) is summed again over its
// own keys alone, without the matrix instructions.
//
// What bounds it: few units (2048 tokens in 5 prompts and 16 heads are 176, of one to nine tiles each, on 148 SMs), and in a unit the way
// S -> softmax -> P V.  Microseconds a layer, 16 heads on rank 512, the folded form (mma.sync) -> here: prompts of 64, 422, 91, 388
// and 1083 tokens: attention 264 -> 27, all kernels of four layers 3286 -> 2230; 32 prompts of 64 tokens: attention 81 -> 19.  Whole pass of
// four layers of the first 3.34 -> 2.56 ms, its error against 64 bits 0.0058 -> 0.0055.
//
// No wait is unbounded: after about two seconds a role gives up, raises the word that gemm_pair_failed() looks at and leaves;
// copies and MMAs in flight land first and TMEM is freed on every path.
#include <algorithm>

#include "attn_tc.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace tgis {
namespace {

constexpr int LH_THREADS = 384;                          // warps 0..3 softmax of accumulator 0, 4..7 of 1, 8 copies, 9 MMAs, 10 and 11 idle
constexpr int LH_REGS_SOFTMAX = 208, LH_REGS_OTHER = 88; // 256 x 208 + 128 x 88 = 384 x 168, what the launch gives every thread
constexpr int LH_KV = 128, LH_CHUNK = 128 * 128;         // keys of a tile; bytes of 64 dims of 128 rows
constexpr int LH_QC = (LATENT_HEAD_DIM + LATENT_HEAD_ROT) / 64, LH_VC = LATENT_HEAD_VDIM / 64, LH_KC = LATENT_HEAD_DIM / 64;
constexpr int LH_QK = LATENT_HEAD_DIM + LATENT_HEAD_ROT;
constexpr int LH_Q_BYTES = LH_QC * LH_CHUNK, LH_V_BYTES = LH_VC * LH_CHUNK;
constexpr size_t LH_SMEM = 2 * LH_Q_BYTES + 2 * LH_Q_BYTES + LH_V_BYTES + 1024 + 256;   // Q, two K tiles, one V tile, barriers
static_assert(LH_SMEM <= 227 * 1024 && LATENT_HEAD_ROT == 64 && LATENT_HEAD_VDIM == 128, "layout");
constexpr float LH_SLACK = 8.f, LH_LOG2E = 1.4426950408889634f;

struct HeadsArgs {
  const __nv_bfloat16 *q, *kv, *rot;   // [T][H][192]; [keys][H][128] | [H][128]; [keys][64]
  const float *gate, *sink;            // [T][H] or nullptr; [H] or nullptr
  const LatentUnit* units;
  __nv_bfloat16* out;                  // [T][H][128]
  int n_units, H, window;
  float sl2;                           // |scale| * log2(e)
  uint32_t minus;                      // scale < 0: bit "negate A" of the score products' descriptor
  int* err;
};

struct Unit : LatentUnit {
  int j0, n_kt, head;   // tiles j0 .. n_kt - 1
  bool two;             // the second accumulator has rows
};
// units of CTA b: b, 2 n - 1 - b, 2 n + b, ... (n CTAs): with the longest first, every CTA's share is about the same
struct UnitIter {
  const HeadsArgs& a;
  int round = 0;
  __device__ explicit UnitIter(const HeadsArgs& a_) : a(a_) {}
  __device__ bool next(Unit& u) {
    const int n = gridDim.x, i = round * n + ((round & 1) ? n - 1 - (int)blockIdx.x : (int)blockIdx.x);
    if (i >= a.n_units) return false;   // the last round is the only one that is not full
    const int4 v = __ldg(reinterpret_cast<const int4*>(a.units) + i / a.H);
    static_cast<LatentUnit&>(u) = LatentUnit{v.x, v.y, v.z, v.w};
    u.head = i % a.H;
    u.j0 = a.window > 0 ? max(0, u.pos0 - a.window + 1) / LH_KV : 0;
    u.n_kt = (u.pos0 + u.rows - 1) / LH_KV + 1;
    u.two = u.rows > 128;
    ++round;
    return true;
  }
};

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float dot8(const uint4& x, const uint4& k, float s) {
  s = fmaf(bf_lo(x.x), bf_lo(k.x), s); s = fmaf(bf_hi(x.x), bf_hi(k.x), s);
  s = fmaf(bf_lo(x.y), bf_lo(k.y), s); s = fmaf(bf_hi(x.y), bf_hi(k.y), s);
  s = fmaf(bf_lo(x.z), bf_lo(k.z), s); s = fmaf(bf_hi(x.z), bf_hi(k.z), s);
  s = fmaf(bf_lo(x.w), bf_lo(k.w), s); s = fmaf(bf_hi(x.w), bf_hi(k.w), s);
  return s;
}
__device__ __forceinline__ const __nv_bfloat16* value_of(const HeadsArgs& a, const Unit& u, int key) {
  return a.kv + (size_t)(u.key0 + key) * a.H * (LATENT_HEAD_DIM + LATENT_HEAD_VDIM) + (size_t)a.H * LATENT_HEAD_DIM + u.head * LATENT_HEAD_VDIM;
}
// One row by a warp, in the order of the keys: lane = key for the scores (twice), lane = four dims for the values, whose weights sum to
// one (less the sink's), so that no sum passes the largest value.
__device__ __forceinline__ void attend_row(const HeadsArgs& a, const Unit& u, int row, int pos) {
  const int lane = (int)lane_id(), lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
  const float sl2 = a.minus != 0 ? -a.sl2 : a.sl2;
  const uint4* q = reinterpret_cast<const uint4*>(a.q + ((size_t)row * a.H + u.head) * LH_QK);
  auto score = [&](int key) {
    if (key < lo || key > pos) return -INFINITY;
    const uint4* k = reinterpret_cast<const uint4*>(a.kv + (size_t)(u.key0 + key) * a.H * (LATENT_HEAD_DIM + LATENT_HEAD_VDIM) + u.head * LATENT_HEAD_DIM);
    const uint4* r = reinterpret_cast<const uint4*>(a.rot + (size_t)(u.key0 + key) * LATENT_HEAD_ROT);
    float s = 0.f;
#pragma unroll 2
    for (int c = 0; c < LATENT_HEAD_DIM / 8; ++c) s = dot8(q[c], k[c], s);
#pragma unroll 2
    for (int c = 0; c < LATENT_HEAD_ROT / 8; ++c) s = dot8(q[LATENT_HEAD_DIM / 8 + c], r[c], s);
    return s * sl2;
  };
  float m = -INFINITY, l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int b = lo / 32 * 32; b <= pos; b += 32) {   // maximum and sum of the lane's keys
    const float x = score(b + lane), top = fmaxf(m, x);
    if (top > -INFINITY) l = l * ex2(m - top) + ex2(x - top);
    m = top;
  }
  float ref = m;
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) ref = fmaxf(ref, __shfl_xor_sync(0xffffffffu, ref, i));
  l *= ex2(m - ref);
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) l += __shfl_xor_sync(0xffffffffu, l, i);
  if (a.sink != nullptr) l += ex2(a.sink[u.head] * LH_LOG2E - ref);
  const float inv = 1.f / l * (a.gate != nullptr ? a.gate[(size_t)row * a.H + u.head] : 1.f);
#pragma unroll 1
  for (int b = lo / 32 * 32; b <= pos; b += 32) {
    const float p = ex2(score(b + lane) - ref) * inv;
    const int t0 = max(0, lo - b), t1 = min(32, pos - b + 1);   // (hidden keys are not touched)
#pragma unroll 4
    for (int t = t0; t < t1; ++t) {
      const float w = __shfl_sync(0xffffffffu, p, t);
      const uint2 v = *reinterpret_cast<const uint2*>(value_of(a, u, b + t) + lane * 4);
      o[0] = fmaf(w, bf_lo(v.x), o[0]); o[1] = fmaf(w, bf_hi(v.x), o[1]);
      o[2] = fmaf(w, bf_lo(v.y), o[2]); o[3] = fmaf(w, bf_hi(v.y), o[3]);
    }
  }
  *reinterpret_cast<uint2*>(a.out + ((size_t)row * a.H + u.head) * LATENT_HEAD_VDIM + lane * 4) = make_uint2(cvt2(o[0], o[1]), cvt2(o[2], o[3]));
}

// The CTA's rows that came out with numbers that are not finite, by its softmax warps, which have stored them all.  Where a key that the
// row sees accounts for them they stand: a unit's values are looked through once for the first such key of every dim, so that a
// sequence which has overflowed costs no more than that.  (A row whose window has moved on is summed again in any case.)
__device__ __noinline__ void sum_again(const HeadsArgs& a) {
  const int lane = (int)lane_id();
  auto odd = [](const uint2& w) {   // one bit per number of four
    const uint32_t e = 0x7f80u;
    return ((w.x & e) == e) | ((w.x >> 16 & e) == e) << 1 | ((w.y & e) == e) << 2 | ((w.y >> 16 & e) == e) << 3;
  };
  Unit u;
  for (UnitIter it(a); it.next(u);) {
    int first[4] = {-1, -1, -1, -1};   // of the lane's dims: the first key whose value is not finite (none: behind the last key)
    for (int r = threadIdx.x >> 5; r < u.rows; r += 8) {
      const int row = u.row0 + r, pos = u.pos0 + r;
      const int mine = odd(*reinterpret_cast<const uint2*>(a.out + ((size_t)row * a.H + u.head) * LATENT_HEAD_VDIM + lane * 4));
      if (!__any_sync(0xffffffffu, mine != 0)) continue;
      if (first[0] < 0) {
        const int n = u.pos0 + u.rows;
        int seen = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) first[e] = n;
        for (int b = u.j0 * LH_KV; b < n && !__all_sync(0xffffffffu, seen == 15); b += 32) {
#pragma unroll 4
          for (int k = b; k < min(b + 32, n); ++k) {
            const int now = odd(*reinterpret_cast<const uint2*>(value_of(a, u, k) + lane * 4)) & ~seen;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (now >> e & 1) first[e] = k;
            seen |= now;
          }
        }
      }
      int hidden = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) hidden |= (first[e] > pos || (a.window > 0 && first[e] <= pos - a.window)) << e;
      if (__any_sync(0xffffffffu, (mine & hidden) != 0)) attend_row(a, u, row, pos);
    }
  }
}

__global__ void __launch_bounds__(LH_THREADS, 1)
attn_heads_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kvmap, const __grid_constant__ CUtensorMap rmap,
                  const __grid_constant__ HeadsArgs a) {
  constexpr int WARP_COPY = 8, WARP_MMA = 9;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;                        // [2 accumulators][3 chunks]
  uint8_t* k_s = q_s + 2 * LH_Q_BYTES;        // [2 tiles][3 chunks]
  uint8_t* v_s = k_s + 2 * LH_Q_BYTES;        // [2 chunks]
  uint64_t* q_full = reinterpret_cast<uint64_t*>(v_s + LH_V_BYTES);
  uint64_t* q_empty = q_full + 1;
  uint64_t* k_full = q_empty + 1;             // [2]
  uint64_t* k_empty = k_full + 2;             // [2]
  uint64_t* v_full = k_empty + 2;
  uint64_t* v_empty = v_full + 1;
  uint64_t* s_full = v_empty + 1;             // [2]
  uint64_t* p_full = s_full + 2;              // [2]
  uint64_t* o_full = p_full + 2;              // [2]
  uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_base_smem + 1);
  volatile int* redo = gave_up + 1;           // rows of the CTA have to be summed again

  const int warp = threadIdx.x >> 5, lane = (int)lane_id();
  UnitIter it(a);   // (the units are written by the host before the step)
  if (warp == WARP_MMA) {
    if (elect_one()) {
      mbar_init(q_full, 1);
      mbar_init(q_empty, 1);
      mbar_init(v_full, 1);
      mbar_init(v_empty, 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&k_full[i], 1);
        mbar_init(&k_empty[i], 1);
        mbar_init(&s_full[i], 1);
        mbar_init(&p_full[i], 4);
        mbar_init(&o_full[i], 1);
      }
      *gave_up = 0;
      *redo = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc<512>(tmem_base_smem);
  }
  if (warp == WARP_COPY && lane == 0) {
    tma_prefetch_desc(&qmap);
    tma_prefetch_desc(&kvmap);
    tma_prefetch_desc(&rmap);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_smem;   // [S0 | S1 | O0 | O1], 128 columns each
  griddep_launch();
  Unit u;
  bool ok = true;
  if (warp >= WARP_COPY) {
    set_regs<LH_REGS_OTHER, false>();
    if (warp == WARP_COPY) {
      // ===================== copies =====================
      int kst = 0;
      uint32_t kph = 1, vph = 1, qph = 1;   // the first pass over a ring finds it empty
      griddep_wait();   // q, keys and values
      while (ok && it.next(u)) {
        ok = __all_sync(0xffffffffu, bounded_wait(q_empty, qph, a.err));
        if (!ok) break;
        qph ^= 1;
        if (lane == 0) {
          const int groups = u.two ? 2 : 1;
          mbar_arrive_expect_tx(q_full, (uint32_t)(groups * LH_Q_BYTES));
          for (int g = 0; g < groups; ++g)
            for (int c = 0; c < LH_QC; ++c)
              tma_load_2d(&qmap, q_full, q_s + g * LH_Q_BYTES + c * LH_CHUNK, u.head * LH_QK + c * 64, u.row0 + g * 128);
        }
        for (int j = u.j0; j < u.n_kt; ++j) {
          ok = __all_sync(0xffffffffu, bounded_wait(&k_empty[kst], kph, a.err));
          if (!ok) break;
          if (lane == 0) {
            mbar_arrive_expect_tx(&k_full[kst], (uint32_t)LH_Q_BYTES);
            for (int c = 0; c < LH_KC; ++c)
              tma_load_2d(&kvmap, &k_full[kst], k_s + kst * LH_Q_BYTES + c * LH_CHUNK, u.head * LATENT_HEAD_DIM + c * 64, u.key0 + j * LH_KV);
            tma_load_2d(&rmap, &k_full[kst], k_s + kst * LH_Q_BYTES + LH_KC * LH_CHUNK, 0, u.key0 + j * LH_KV);
          }
          __syncwarp();
          if (++kst == 2) kst = 0, kph ^= 1;
          ok = __all_sync(0xffffffffu, bounded_wait(v_empty, vph, a.err));
          if (!ok) break;
          if (lane == 0) {
            mbar_arrive_expect_tx(v_full, (uint32_t)LH_V_BYTES);
            for (int c = 0; c < LH_VC; ++c)
              tma_load_2d(&kvmap, v_full, v_s + c * LH_CHUNK, a.H * LATENT_HEAD_DIM + u.head * LATENT_HEAD_VDIM + c * 64, u.key0 + j * LH_KV);
          }
          __syncwarp();
          vph ^= 1;
        }
      }
    } else if (warp == WARP_MMA) {
      // ===================== MMAs =====================
      int kst = 0;
      uint32_t kph = 0, vph = 0, qph = 0, pph[2] = {0, 0};
      const uint32_t idesc_s = make_idesc_bf16(128, LH_KV) | a.minus, idesc_pv = make_idesc_bf16(128, LATENT_HEAD_VDIM) | (1u << 16);   // (V has its dims contiguous)
      auto scores = [&](int g) {
        const uint32_t q = smem_u32(q_s + g * LH_Q_BYTES), k = smem_u32(k_s + kst * LH_Q_BYTES);
#pragma unroll
        for (int ks = 0; ks < LH_QK / 16; ++ks)
          tc_mma_f16(tmem_base + g * 128, make_smem_desc_sw128(q + (ks >> 2) * LH_CHUNK + (ks & 3) * 32),
                     make_smem_desc_sw128(k + (ks >> 2) * LH_CHUNK + (ks & 3) * 32), idesc_s, ks > 0);
        tc_commit(&s_full[g]);
      };
      auto values = [&](int g, bool first) {
        const uint32_t v = smem_u32(v_s);
#pragma unroll
        for (int ks = 0; ks < LH_KV / 16; ++ks)
          mma_ts(tmem_base + 256 + g * 128, tmem_base + g * 128 + ks * 8, smem_desc(v + ks * 2048, LH_CHUNK, 1024, 2), idesc_pv, !(first && ks == 0));
      };
      while (ok && it.next(u)) {
        const int groups = u.two ? 2 : 1;
        ok = __all_sync(0xffffffffu, bounded_wait(q_full, qph, a.err) && bounded_wait(&k_full[kst], kph, a.err));
        if (!ok) break;
        qph ^= 1;
        tc_fence_after();
        if (elect_one()) {
          for (int g = 0; g < groups; ++g) scores(g);
          tc_commit(&k_empty[kst]);
          if (u.j0 + 1 == u.n_kt) tc_commit(q_empty);
        }
        __syncwarp();
        if (++kst == 2) kst = 0, kph ^= 1;
        for (int j = u.j0; j < u.n_kt && ok; ++j) {
          const bool more = j + 1 < u.n_kt;
          ok = __all_sync(0xffffffffu, bounded_wait(v_full, vph, a.err));
          for (int g = 0; g < groups && ok; ++g) {
            ok = __all_sync(0xffffffffu, bounded_wait(&p_full[g], pph[g], a.err) && (g > 0 || !more || bounded_wait(&k_full[kst], kph, a.err)));
            if (!ok) break;
            pph[g] ^= 1;
            tc_fence_after();
            if (elect_one()) {
              const bool last = g == groups - 1;
              values(g, j == u.j0);
              if (last) tc_commit(v_empty);
              if (more) scores(g);
              if (last) {
                if (more) tc_commit(&k_empty[kst]);
                if (j + 2 == u.n_kt) tc_commit(q_empty);
              }
              if (!more) tc_commit(&o_full[g]);
            }
            __syncwarp();
          }
          vph ^= 1;
          if (more && ++kst == 2) kst = 0, kph ^= 1;
        }
      }
    }
  } else {
    // ===================== softmax: thread = row =====================
    set_regs<LH_REGS_SOFTMAX, true>();
    const int g = warp >> 2, r = g * 128 + (warp & 3) * 32 + lane;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_t = tmem_base + g * 128 + lanes, o_t = tmem_base + 256 + g * 128 + lanes;
    const uint64_t sl2_2 = pack2(a.sl2, a.sl2);
    uint32_t sph = 0, oph = 0;
    griddep_wait();   // `out` may still be read
    while (ok && it.next(u)) {
      if (g == 1 && !u.two) continue;
      const int pos = u.pos0 + r, pos_lo = pos - lane;   // (a row's own, and its warp's first)
      float m = 0.f, l = 0.f;
      for (int j = u.j0; j < u.n_kt; ++j) {
        const int lim = pos - j * LH_KV;   // last column this row sees
        const int low = a.window > 0 ? lim - a.window + 1 : 0;   // ... and the first
        const bool mask = j * LH_KV + LH_KV - 1 > pos_lo || (a.window > 0 && j * LH_KV <= pos_lo + 31 - a.window);
        ok = __all_sync(0xffffffffu, bounded_wait(&s_full[g], sph, a.err));
        if (!ok) break;
        sph ^= 1;
        tc_fence_after();
        uint32_t s[LH_KV];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_x32(s_t + c * 32, s + c * 32);
        tmem_ld_wait();
        if (mask) {
#pragma unroll
          for (int i = 0; i < LH_KV; ++i)
            if (i > lim || i < low) s[i] = __float_as_uint(-INFINITY);
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < LH_KV; i += 2) mx[i >> 5] = fmaxf(mx[i >> 5], fmaxf(__uint_as_float(s[i]), __uint_as_float(s[i + 1])));
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.sl2;
        if (j == u.j0) {
          m = top;
        } else if (__any_sync(0xffffffffu, top > m + LH_SLACK)) {
          // the products that wrote O retired before these scores did
          const float f = top > m + LH_SLACK ? ex2(m - top) : 1.f;
          if (top > m + LH_SLACK) m = top;
          l *= f;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(o_t + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
            tmem_st_x16(o_t + c * 16, o);
          }
        }
        const float ref = m == -INFINITY ? 0.f : m;   // (no score above -inf so far: every probability is 0, not the NaN of inf - inf)
        const uint64_t neg_m = pack2(-ref, -ref);
        uint64_t sum0 = 0, sum1 = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t p8[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int col = c * 16 + 2 * i;
            float x, y;
            unpack2(fma2(pack2(__uint_as_float(s[col]), __uint_as_float(s[col + 1])), sl2_2, neg_m), x, y);
            x = ex2(x);
            y = ex2(y);
            const uint64_t p = pack2(x, y);
            if (i & 1) sum1 = add2(sum1, p);
            else sum0 = add2(sum0, p);
            p8[i] = cvt2(x, y);
          }
          tmem_st_x8(s_t + c * 8, p8);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[g]);
        float x, y;
        unpack2(add2(sum0, sum1), x, y);
        l += x + y;
      }
      if (!ok) break;
      ok = __all_sync(0xffffffffu, bounded_wait(&o_full[g], oph, a.err));
      if (!ok) break;
      oph ^= 1;
      tc_fence_after();
      const bool wanted = r < u.rows;
      const size_t at = (size_t)(u.row0 + (wanted ? r : 0)) * a.H + u.head;
      if (a.sink != nullptr) l += ex2(a.sink[u.head] * LH_LOG2E - m);   // (a causal row sees itself: m is a number)
      const float inv = 1.f / l * (a.gate != nullptr ? a.gate[at] : 1.f);
      __nv_bfloat16* dst = a.out + at * LATENT_HEAD_VDIM;
      float odd = 0.f;   // NaN where numbers of the row are not finite (taken eight at a time: all of them at once spill)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld_x32(o_t + c * 32, o);
        tmem_ld_wait();
        if (wanted) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = cvt2(__uint_as_float(o[i * 8 + 2 * k]) * inv, __uint_as_float(o[i * 8 + 2 * k + 1]) * inv);
            float z = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) z += __uint_as_float(o[i * 8 + k]);
            odd = fmaf(z, 0.f, odd);
            *reinterpret_cast<uint4*>(dst + c * 32 + i * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      tc_fence_before();
      if (wanted && l - l == 0.f && odd != 0.f) *redo = 1;
    }
  }
  if (!ok && lane == 0) *gave_up = 1;
  tc_fence_before();
  __syncthreads();
  // rows whose numbers may come from keys that they do not see (registers: only the softmax warps have enough)
  if (*redo != 0 && *gave_up == 0 && warp < WARP_COPY) sum_again(a);
  // after a wait that ran out copies and MMAs of the other roles may be in flight; they are done long before this millisecond is over
  if (*gave_up)
    for (const long long t0 = clock64(); clock64() - t0 < 2000000ll;) {}
  __syncthreads();
  if (warp == WARP_MMA) {
    tc_fence_after();
    tmem_dealloc<512>(tmem_base);
  }
}

// Blocks 0 .. n_blocks - 1 (of all spans): a cache block's rows to their places among the gathered ones.  Blocks behind them: the rotary part of a
// token's queries turned in place (the arithmetic of latent_q_rope_kernel, rounded to bf16 here).
__global__ void __launch_bounds__(256)
latent_rows_kernel(const __nv_bfloat16* __restrict__ cache, const LatentSpan* __restrict__ spans, int n_blocks, const int32_t* __restrict__ block_table,
                   int bt_stride, int kv_rank, __nv_bfloat16* __restrict__ rows,
                   __nv_bfloat16* __restrict__ rot, __nv_bfloat16* __restrict__ q, LatentGeom g, const int32_t* __restrict__ positions,
                   const float* __restrict__ cos_sin) {
  griddep_launch();
  griddep_wait();
  if ((int)blockIdx.x < n_blocks) {
    int b = blockIdx.x;
    LatentSpan sp = spans[0];
    while (b * KV_BLOCK >= sp.n) {
      b -= (sp.n + KV_BLOCK - 1) / KV_BLOCK;
      sp = *++spans;
    }
    const int n = min(KV_BLOCK, sp.n - b * KV_BLOCK), row = sp.row + b * KV_BLOCK;
    const int per = (kv_rank + LATENT_HEAD_ROT) / 8, plain = kv_rank / 8;
    const uint4* from = reinterpret_cast<const uint4*>(cache) + (size_t)block_table[(size_t)sp.block_row * bt_stride + sp.first / KV_BLOCK + b] * KV_BLOCK * per;
    for (int e = threadIdx.x; e < n * per; e += blockDim.x) {
      const int r = e / per, c = e - r * per;
      const uint4 v = from[e];
      if (c < plain) reinterpret_cast<uint4*>(rows)[(size_t)(row + r) * plain + c] = v;
      else reinterpret_cast<uint4*>(rot)[(size_t)(row + r) * (LATENT_HEAD_ROT / 8) + c - plain] = v;
    }
    return;
  }
  const int t = blockIdx.x - n_blocks, half = g.rot_dims / 2;
  const float* cs = cos_sin + (size_t)positions[t] * g.rot_dims;
  for (int e = threadIdx.x; e < g.heads * half; e += blockDim.x) {
    const int h = e / half, j = e - h * half;
    __nv_bfloat16* v = q + ((size_t)t * g.heads + h) * LH_QK + LATENT_HEAD_DIM;
    const int i0 = g.interleaved ? 2 * j : j, i1 = g.interleaved ? 2 * j + 1 : j + half;
    const float x = __bfloat162float(v[i0]), y = __bfloat162float(v[i1]), c = cs[j], s = cs[half + j];
    v[i0] = __float2bfloat16_rn(x * c - y * s);
    v[i1] = __float2bfloat16_rn(y * c + x * s);
  }
}

}  // namespace

bool latent_heads_takes(const LatentGeom& g, int dtype) {
  return dtype == DT_BF16 && g.dim == LATENT_HEAD_DIM && g.rot_dim == LATENT_HEAD_ROT && g.vdim == LATENT_HEAD_VDIM && g.kv_rank % 64 == 0 &&
         g.kv_rank >= 64 && g.rot_dims <= LATENT_HEAD_ROT && g.rot_dims % 2 == 0;
}

int latent_units_build(LatentUnit* units, const AttnSeq& q, int first, int key0) {
  int n = 0;
  for (int q0 = 0; q0 < q.q_len; q0 += 256)
    units[n++] = LatentUnit{q.q_start + q0, std::min(256, q.q_len - q0), q.kv_len - q.q_len + q0 - first, key0};
  return n;
}
void latent_units_sort(LatentUnit* units, int n) {
  std::stable_sort(units, units + n, [](const LatentUnit& x, const LatentUnit& y) { return (x.pos0 + x.rows - 1) / LH_KV > (y.pos0 + y.rows - 1) / LH_KV; });
}

cudaError_t latent_rows_launch(const void* cache, const LatentSpan* spans, int n_blocks, const int32_t* block_table, int bt_stride, void* rows, void* rot,
                               void* q, const LatentGeom& g, const int32_t* positions, const float* cos_sin, int T, cudaStream_t stream) {
  if (n_blocks + T <= 0) return cudaSuccess;
  if (!latent_heads_takes(g, DT_BF16)) return cudaErrorInvalidValue;
  return launch_k(latent_rows_kernel, dim3(n_blocks + T), dim3(256), 0, stream, (const __nv_bfloat16*)cache, spans, n_blocks, block_table, bt_stride, g.kv_rank, (__nv_bfloat16*)rows,
                  (__nv_bfloat16*)rot, (__nv_bfloat16*)q, g, positions, cos_sin);
}

cudaError_t latent_heads_launch(const void* q, int T, const void* kv, const void* rot, int n_keys, const LatentUnit* units, int n_units, const float* gate,
                                void* out, const LatentGeom& g, int num_sms, cudaStream_t stream) {
  if (n_units <= 0) return cudaSuccess;
  if (!latent_heads_takes(g, DT_BF16) || n_keys <= 0) return cudaErrorInvalidValue;
  HeadsArgs a{};
  cudaError_t e = gemm_pair_word(&a.err);
  if (e != cudaSuccess) return e;
  a.q = (const __nv_bfloat16*)q; a.kv = (const __nv_bfloat16*)kv; a.rot = (const __nv_bfloat16*)rot;
  a.gate = gate; a.sink = g.sink; a.units = units; a.out = (__nv_bfloat16*)out;
  a.n_units = n_units * g.heads; a.H = g.heads; a.window = g.window;
  a.sl2 = g.scale != 0.f ? fabsf(g.scale) * LH_LOG2E : 1e-30f;   // hidden scores are -inf before they are scaled
  a.minus = g.scale < 0.f ? 1u << 13 : 0u;
  const int kv_cols = g.heads * (LATENT_HEAD_DIM + LATENT_HEAD_VDIM);
  CUtensorMap qm, km, rm;
  if (make_tmap_bf16_2d(&qm, q, T, (uint64_t)g.heads * LH_QK, (uint64_t)g.heads * LH_QK, 128, 64) != 0 ||
      make_tmap_bf16_2d(&km, kv, n_keys, kv_cols, kv_cols, LH_KV, 64) != 0 ||
      make_tmap_bf16_2d(&rm, rot, n_keys, LATENT_HEAD_ROT, LATENT_HEAD_ROT, LH_KV, 64) != 0)
    return cudaErrorInvalidValue;
  static const cudaError_t attr = cudaFuncSetAttribute(attn_heads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LH_SMEM);
  if (attr != cudaSuccess) return attr;
  return launch_k(attn_heads_kernel, dim3(std::min(a.n_units, num_sms)), dim3(LH_THREADS), LH_SMEM, stream, qm, km, rm, a);
}

}  // namespace tgis
