// ONE fused TGIS sampling kernel: everything between the lm_head logits and the (token, logprob, rank, top-n) record.
//
// It replaces ~30 small launches + a per-request Python loop in the reference stack:
//   reference-owned : tgis_utils/logits_processors.py:24-47  ExpDecayLengthPenaltyWarper      (R7)
//                     tgis_utils/logits_processors.py:7-21   TypicalLogitsWarperWrapper       (R8)
//                       -> hf generation/logits_process.py:836-856
//   vllm 0.22       : v1/sample/sampler.py:67-144 (raw log-softmax, min_tokens, penalties, greedy/temperature,
//                     top-k/top-p, exponential-race sampling, gather_logprobs + rank)         (S1-S8)
// Contract order per row: raw log-softmax -> typical-p -> ExpDecay(EOS) -> min_tokens(EOS)
// -> repetition penalty -> greedy argmax | temperature -> top-k -> top-p -> sample -> logprob / rank / top-n (raw).
//
// Shape of the problem: a [rows, V=128256] scan with integer-ish selection work; a sampling row needs several passes of
// 50-100 instructions per element, which is ISSUE bound on one SM.  So a row is owned by a thread-block CLUSTER of up to 8 CTAs x
// 1024 threads: each scans its part of the vocabulary, block results are exchanged through distributed shared memory and combined
// in a fixed order (deterministic).  The row is read from HBM once and stays in shared memory or the L2 for the selection passes
// (radix-select thresholds instead of the reference's full sorts).  Every sweep takes eight entries per thread and 16-byte load.
//   first sweep   32 entries a thread at a time: their maximum, then exponentials that do not wait for one another (an online
//                 maximum per entry was a chain of a branch and an exponential each); behind typical-p the entropy's sum too
//   reductions    maximum, sums and best entry in one; an exchange is one 16-byte read per lane and shuffles
//   selections    (typical-p, top-k, top-p) one sweep over steps of a 32nd of an octave, one that lists the selected step's entries, then
//                 parts of a step and radix rounds over the list
//   race          behind typical-p over the list of what is left; in flat rows over kept processed logits, two logarithms only
//                 for entries that 1 - u cannot rule out
//   rank, top-n   one sweep and one exchange, the slices' lists ordered by eight threads a candidate
// Measured, 128256 bf16 logits with top-5, microseconds, with the online maximum, an exchange for each part, clusters by SM count and four
// radix rounds over leading bits -> here: greedy 19.7 -> 14 (1 row), 39 -> 15 (16), 22 -> 15 (32), 36 -> 29 (80), 73 -> 55 (150); typical-p
// 44 -> 29 (1), 88 -> 38 (16), 61 -> 38 (32), 157 -> 91 (80), 312 -> 178 (150); flat rows 62 -> 41 (1), 286 -> 173 (80); top-k with top-p
// 61 -> 42 (1), 238 -> 133 (80).  Warp instructions of 96 rows, millions (profiles/work_ncu.csv): greedy 19 -> 16, flat typical-p 152 -> 92.
#include <cooperative_groups.h>

#include <type_traits>

#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace cg = cooperative_groups;

namespace tgis {

TGIS_STL_DEFINE(sampler)

constexpr int SAMP_THREADS = 1024;
constexpr int SAMP_WARPS = SAMP_THREADS / 32;
constexpr int SAMP_LIST = SAMP_THREADS;      // entries a race or a top-n list holds
constexpr int SAMP_FEW = 3 * SAMP_THREADS;   // ... a selection's list
constexpr float SAMP_FLAT = 7.f;  // nats: as spread as over 1100 entries, more than the list of a row's only CTA holds (of 2 to 8 CTAs: 2048 to 8192)
constexpr float SAMP_FIX = 1073741824.0f;  // 2^30: probabilities are accumulated as fixed-point integers (see below)

// LT = logits element type: __nv_bfloat16 on the product path (vLLM's lm_head emits model-dtype logits and the sampler
// casts them to fp32: vllm v1/sample/sampler.py:91 -- every bf16 value is exactly representable), float for the
// kernel-level golden tests (fp32 fixtures generated from the reference's own code).
template <class LT>
struct RowCtx {
  const LT* x;             // raw logits
  const LT* xc;            // this CTA's slice staged in shared memory by pass 1 (xc[i - lo]), or nullptr
  int V;
  int lo, hi;              // this CTA's slice of the vocabulary (multiples of 8)
  const uint32_t* seen;    // bitmap of prompt U output tokens (may be null)
  const uint32_t* allow;   // guided decoding: bit i set = token i allowed this step (null: unconstrained).  A cleared bit
                           // turns the RAW logit into -inf before anything else looks at it, which is where vLLM applies
                           // its grammar bitmask (v1/worker/gpu_model_runner.py apply_grammar_bitmask, before the sampler)
  SampleRow p;
  float lenfac_m1;         // (float)(decay^n - 1), 0 => inactive
  bool mask_eos;           // min_tokens not reached
  // typical-p state
  bool typical;
  float raw_max, raw_logz, ent, typ_thr;
};

__device__ __forceinline__ float lt2f(float v) { return v; }
__device__ __forceinline__ float lt2f(__nv_bfloat16 v) { return __bfloat162float(v); }
// entry i of this CTA's slice [lo, hi): from the shared-memory copy when the slice was staged (every pass after the first
// then costs shared-memory latency instead of an L2 round trip per dependent load)
template <class LT>
__device__ __forceinline__ bool is_allowed(const RowCtx<LT>& c, int i) {
  return c.allow == nullptr || ((c.allow[i >> 5] >> (i & 31)) & 1u);
}
// any entry of the row (global memory)
template <class LT>
__device__ __forceinline__ float load_x_any(const RowCtx<LT>& c, int i) {
  return is_allowed(c, i) ? lt2f(c.x[i]) : -INFINITY;
}
// (the staged copy already carries the -inf of disallowed tokens: pass 1 masks before it stores)
template <class LT>
__device__ __forceinline__ float load_x(const RowCtx<LT>& c, int i) {
  return c.xc != nullptr ? lt2f(c.xc[i - c.lo]) : load_x_any(c, i);
}
__device__ __forceinline__ void store_x8(float* dst, const float (&v)[8]) {
  *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store_x8(__nv_bfloat16* dst, const float (&v)[8]) {
  uint4 r;
  uint32_t* w = &r.x;
#pragma unroll
  for (int e = 0; e < 4; ++e) w[e] = (__float_as_uint(v[2 * e]) >> 16) | (__float_as_uint(v[2 * e + 1]) & 0xffff0000u);
  *reinterpret_cast<uint4*>(dst) = r;  // exact: the values came from bf16
}
// 8 consecutive logits (i0 % 8 == 0) as fp32
__device__ __forceinline__ void load_x8(const float* x, int i0, float (&o)[8]) {
  const float4 ra = *reinterpret_cast<const float4*>(x + i0);
  const float4 rb = *reinterpret_cast<const float4*>(x + i0 + 4);
  o[0] = ra.x; o[1] = ra.y; o[2] = ra.z; o[3] = ra.w; o[4] = rb.x; o[5] = rb.y; o[6] = rb.z; o[7] = rb.w;
}
__device__ __forceinline__ void load_x8(const __nv_bfloat16* x, int i0, float (&o)[8]) {
  const uint4 r = *reinterpret_cast<const uint4*>(x + i0);
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    o[2 * e] = __uint_as_float(w[e] << 16);
    o[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
  }
}

// eight bits of a token bitmap from entry i0 on (i0 % 8 == 0)
__device__ __forceinline__ uint32_t bits8(const uint32_t* map, int i0) { return (map[i0 >> 5] >> (i0 & 31)) & 0xffu; }
// eight entries of this CTA's slice (i0 % 8 == 0, i0 + 8 <= hi), masked
template <class LT>
__device__ __forceinline__ void load_slice8(const RowCtx<LT>& c, int i0, float (&o)[8]) {
  if (c.xc != nullptr) {
    load_x8(c.xc, i0 - c.lo, o);
    return;
  }
  load_x8(c.x, i0, o);
  if (c.allow != nullptr) {
    const uint32_t bits = bits8(c.allow, i0);
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (!((bits >> e) & 1u)) o[e] = -INFINITY;
  }
}

// processed logits (before temperature) of the entries i0 .. i0 + 7, in place of their raw values
template <class LT>
__device__ __forceinline__ void process8(const RowCtx<LT>& c, int i0, float (&v)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (c.typical) {
      const float lp = (v[e] - c.raw_max) - c.raw_logz;
      const float s = fabsf((-lp) - c.ent);
      if (s > c.typ_thr) v[e] = -INFINITY;
    }
    if (i0 + e == c.p.eos_id) {
      if (c.lenfac_m1 != 0.f && isfinite(v[e])) v[e] = __fadd_rn(v[e], __fmul_rn(fabsf(v[e]), c.lenfac_m1));
      if (c.mask_eos) v[e] = -INFINITY;
    }
  }
  const uint32_t seen = c.seen != nullptr ? bits8(c.seen, i0) : 0u;
  if (seen != 0) {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if ((seen >> e) & 1u) v[e] = (v[e] > 0.f) ? __fdiv_rn(v[e], c.p.rep_penalty) : __fmul_rn(v[e], c.p.rep_penalty);
  }
}

// ---------------------------------------------------------------- block reductions (result in every thread)
// maximum m, sum of e^(x - m) and, for the entropy, sum of (x - m) e^(x - m)
struct MaxSum {
  float m, s, w;
};
// ... as they are against a larger maximum
__device__ __forceinline__ MaxSum ms_against(MaxSum t, float m) {
  if (t.m == -INFINITY) return {m, 0.f, 0.f};
  const float d = t.m - m, f = expf(d);
  return {m, t.s * f, f * (t.w + d * t.s)};
}
// argmax with lowest-index tie break (torch.argmax semantics relied on by greedy parity)
struct ValIdx {
  float v;
  int i;
};
__device__ __forceinline__ ValIdx vi_better(ValIdx a, ValIdx b) {
  if (b.i < 0) return a;
  if (a.i < 0) return b;
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ __forceinline__ ValIdx warp_argmax(ValIdx v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ValIdx t{__shfl_xor_sync(0xffffffffu, v.v, o), __shfl_xor_sync(0xffffffffu, v.i, o)};
    v = vi_better(v, t);
  }
  return v;
}
__device__ ValIdx block_argmax(ValIdx v, float* redf, int* redi) {
  v = warp_argmax(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) {
    redf[w] = v.v;
    redi[w] = v.i;
  }
  __syncthreads();
  return warp_argmax(ValIdx{redf[l], redi[l]});
}
// these together with the best entry: every sum is brought to its warp's and then to the block's maximum once
struct MaxSumBest {
  MaxSum ms;
  ValIdx best;
};
__device__ __forceinline__ MaxSumBest warp_maxsum_best(MaxSumBest t) {
  float m = t.ms.m;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  t.ms = ms_against(t.ms, m);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    t.ms.s += __shfl_xor_sync(0xffffffffu, t.ms.s, o);
    t.ms.w += __shfl_xor_sync(0xffffffffu, t.ms.w, o);
    const ValIdx b{__shfl_xor_sync(0xffffffffu, t.best.v, o), __shfl_xor_sync(0xffffffffu, t.best.i, o)};
    t.best = vi_better(t.best, b);
  }
  return t;
}
struct RedBest {
  float m, s, w, v;
  int i;
};
__device__ __forceinline__ MaxSumBest block_maxsum_best(MaxSumBest t, RedBest* red /*[SAMP_WARPS]*/) {
  t = warp_maxsum_best(t);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = RedBest{t.ms.m, t.ms.s, t.ms.w, t.best.v, t.best.i};
  __syncthreads();
  static_assert(SAMP_WARPS == 32, "a lane per warp");
  const RedBest r = red[l];
  return warp_maxsum_best(MaxSumBest{{r.m, r.s, r.w}, {r.v, r.i}});
}
__device__ float block_sumf(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float r = red[l];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}
__device__ int block_sumi(int v, int* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  int r = red[l];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}

// ---------------------------------------------------------------- cluster exchange (ncl CTAs, combined in rank order)
// Every exchange costs ONE cluster barrier: the 4-word slots rotate (exchange e uses slot e & 1), and a CTA can only
// overwrite slot e & 1 for exchange e + 2 after passing the barrier of exchange e + 1, which every peer reaches only
// after it has finished reading exchange e.  The histograms of the radix selects rotate the same way.  A launch with
// one CTA per row (ncl == 1) degenerates to block barriers.
struct Cl {
  int ncl, rank;
  int xe, he;  // exchange / histogram round counters
  __device__ void sync() const {
    if (ncl > 1) cg::this_cluster().sync();
    else __syncthreads();
  }
};
template <class T>
__device__ __forceinline__ T dsmem_read(const Cl& c, T* local, int rank) {
  return c.ncl > 1 ? *cg::this_cluster().map_shared_rank(local, rank) : *local;
}
struct Xch4 {
  float a, b, c, d;
};
// publish this CTA's words (already block-reduced: every thread holds them); lane r of every warp then holds those of rank r
struct XchView {
  float4 mine;
  __device__ Xch4 get(int r) const {
    return Xch4{__shfl_sync(0xffffffffu, mine.x, r), __shfl_sync(0xffffffffu, mine.y, r), __shfl_sync(0xffffffffu, mine.z, r),
                __shfl_sync(0xffffffffu, mine.w, r)};
  }
};
__device__ XchView cl_publish(Cl& c, float4* xch, Xch4 v) {
  float4* slot = xch + (c.xe & 1);
  ++c.xe;
  if (threadIdx.x == 0) *slot = make_float4(v.a, v.b, v.c, v.d);
  c.sync();
  const int lane = threadIdx.x & 31;
  return XchView{dsmem_read(c, slot, lane < c.ncl ? lane : 0)};
}
__device__ float cluster_max(Cl& c, float v, float* red, float4* xch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float m = red[l];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  m = cl_publish(c, xch, Xch4{m, 0.f, 0.f, 0.f}).mine.x;   // (lanes behind the last rank repeat rank 0)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}
__device__ ValIdx cluster_argmax(Cl& c, ValIdx v, float* redf, int* redi, float4* xch) {
  v = block_argmax(v, redf, redi);
  const XchView w = cl_publish(c, xch, Xch4{v.v, __int_as_float(v.i), 0.f, 0.f});
  Xch4 t = w.get(0);
  ValIdx acc{t.a, __float_as_int(t.b)};
  for (int r = 1; r < c.ncl; ++r) {
    t = w.get(r);
    acc = vi_better(acc, ValIdx{t.a, __float_as_int(t.b)});
  }
  return acc;
}
__device__ float cluster_sumf(Cl& c, float v, float* red, float4* xch) {
  v = block_sumf(v, red);
  const XchView w = cl_publish(c, xch, Xch4{v, 0.f, 0.f, 0.f});
  float acc = w.get(0).a;
  for (int r = 1; r < c.ncl; ++r) acc += w.get(r).a;
  return acc;
}

// ---------------------------------------------------------------- radix select helpers
__device__ __forceinline__ uint32_t f2key(float f) {  // order preserving float -> uint
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key2f(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// One radix round shared by the two selects: the CTA's histogram (hist[256], integer bins) is complete; sum the
// cluster's histograms in rank order, then warp 0 scans the 256 bins in parallel (8 per lane + a shuffle prefix).
//   ascending (weighted select): first bin b with  below + sum_{<= b} >= target  (strict: > target); none: last nonempty
//   descending (k-th largest)  : first bin b from the top with  above + sum_{>= b} >= target
// Returns (bin, weight strictly before the bin in scan order, whether any bin has weight) to every thread through bcast[0..2].
template <int BINS>
__device__ void radix_round_pick(const Cl& c, uint32_t* hist, uint32_t* hsum, uint32_t* bcast, uint32_t before,
                                 uint32_t target, bool strict, bool descending) {
  c.sync();  // every CTA's histogram of this round is complete
  if (threadIdx.x < BINS) {
    uint32_t t = 0;
    for (int r = 0; r < c.ncl; ++r) t += dsmem_read(c, hist + threadIdx.x, r);
    hsum[threadIdx.x] = t;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int l = threadIdx.x;
    constexpr int PER = BINS / 32;
    uint32_t h[PER], tot = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int b = descending ? BINS - 1 - (PER * l + j) : PER * l + j;
      h[j] = hsum[b];
      tot += h[j];
    }
    uint32_t incl = tot;  // inclusive prefix over lanes (scan order)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (l >= o) incl += t;
    }
    uint32_t cum = before + incl - tot;  // weight before this lane's first bin
    int sel = -1;
    uint32_t sel_before = 0;
    int last_nonempty = -1;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const uint32_t nc = cum + h[j];
      if (h[j] > 0) last_nonempty = PER * l + j;
      if (sel < 0 && h[j] > 0 && (strict ? (nc > target) : (nc >= target))) {
        sel = PER * l + j;
        sel_before = cum;
      }
      cum = nc;
    }
    const uint32_t hit = __ballot_sync(0xffffffffu, sel >= 0);
    const uint32_t nonempty = __ballot_sync(0xffffffffu, tot > 0);
    int out_sel;
    uint32_t out_before;
    if (hit) {
      const int src = __ffs(hit) - 1;
      out_sel = __shfl_sync(0xffffffffu, sel, src);
      out_before = __shfl_sync(0xffffffffu, sel_before, src);
    } else {
      // rounding: total weight < target -> keep everything: choose the last nonempty bin in scan order
      int ln = last_nonempty;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ln = max(ln, __shfl_xor_sync(0xffffffffu, ln, o));
      out_sel = ln < 0 ? BINS - 1 : ln;
      // weight before that bin: lanes below contribute their totals, the owning lane its bins before it
      uint32_t part = 0;
#pragma unroll
      for (int j = 0; j < PER; ++j)
        if (PER * l + j < out_sel) part += h[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      out_before = before + part;
    }
    if (l == 0) {
      bcast[0] = (uint32_t)(descending ? BINS - 1 - out_sel : out_sel);  // back to a digit value
      bcast[1] = out_before;
      bcast[2] = nonempty;
    }
  }
  __syncthreads();
}

// Adds eight (digit, weight) pairs of every lane to the histogram (weight 0: does not count).  Where the whole warp's 256
// entries share a digit (the leading digits of most rows) one redux and one atomic do, where a lane's eight do one atomic; else every
// entry is a shared-memory atomic of its own, on several copies of the histogram so that lanes of equal digits meet less often.
constexpr int HIST_WORDS = 1024;   // copies of the histogram, as many as fit
template <int BINS>
__device__ __forceinline__ void hist_add8(uint32_t* h, const uint32_t (&digit)[8], const uint32_t (&w)[8]) {
  uint32_t d = 0xffffffffu, sum = 0;
  bool same = true;
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (w[e] > 0) {
      if (d == 0xffffffffu) d = digit[e];
      same &= digit[e] == d;
      sum += w[e];
    }
  const uint32_t have = __ballot_sync(0xffffffffu, d != 0xffffffffu);
  if (have == 0) return;
  const uint32_t d0 = __shfl_sync(0xffffffffu, d, __ffs(have) - 1);
  if (__all_sync(0xffffffffu, same && (d == d0 || d == 0xffffffffu))) {
    const uint32_t all = __reduce_add_sync(0xffffffffu, sum);
    if ((threadIdx.x & 31) == 0) atomicAdd(&h[d0], all);
    return;
  }
  uint32_t* mine = h + (threadIdx.x & (HIST_WORDS / BINS - 1)) * BINS;
  if (same) {
    if (sum > 0) atomicAdd(&mine[d], sum);
    return;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (w[e] > 0) atomicAdd(&mine[digit[e]], w[e]);
}
// a round's histogram: all copies to zero / their sum in the first
__device__ __forceinline__ void hist_clear(uint32_t* h) {
  for (int i = threadIdx.x; i < HIST_WORDS; i += SAMP_THREADS) h[i] = 0u;
  __syncthreads();
}
template <int BINS>
__device__ __forceinline__ void hist_fold(uint32_t* h) {
  __syncthreads();
  if (threadIdx.x < BINS) {
    uint32_t t = h[threadIdx.x];
#pragma unroll
    for (int k = 1; k < HIST_WORDS / BINS; ++k) t += h[k * BINS + threadIdx.x];
    h[threadIdx.x] = t;
  }
}

// The first sweep of a selection sorts by this instead of by leading bits: of a distance >= 0, steps of a 32nd of an octave from 2^-10
// to 2^6 (what lies outside joins the first or the last).  Leading bits of a float are its exponent: two steps of an octave hold nine
// tenths of a flat row, which then was swept three times, with an exponential and an atomic for most entries each time.
constexpr int CODES = 512;
constexpr uint32_t CODE_FIRST = (127 - 10) << 5;   // leading 14 bits of the lowest step
__device__ __forceinline__ uint32_t distance_code(float t) {
  const int c = (int)(__float_as_uint(t) >> 18) - (int)CODE_FIRST;
  return (uint32_t)min(max(c, 0), CODES - 1);
}
// ... and, within a step, by 512 of its parts: the next nine bits; equal parts of the lowest step, which begins at zero; steps of a 512th of
// an octave in the last
__device__ __forceinline__ uint32_t distance_part(float t) {
  const uint32_t b = __float_as_uint(t), c = distance_code(t);
  if (c == 0) return min((uint32_t)(t * 508400.f), (uint32_t)CODES - 1);   // (512 parts of 33 / 32 2^-10)
  if (c == CODES - 1) return min((b >> 14) - ((CODE_FIRST + CODES - 1) << 4), (uint32_t)CODES - 1);
  return (b >> 9) & (CODES - 1);
}

// Smallest key K (ascending) such that  sum_{key_i <= K} w_i  >= target  (strict: > target), or with `descending` the largest with
// sum_{key_i >= K}; if never reached, the last present key.  load(i0, v) -> eight values; (code(v), part(v)), each < CODES, do not fall as
// the key rises; keyf(v) -> uint32 key, wq(v) -> integer weight: integer addition is associative, so the result is the same on every
// cluster size.  Every CTA histograms its slice, the cluster sums the histograms, every CTA runs the same scan: codes over the slice; a
// sweep that lists the entries of the selected code; parts over the list, or, where that has no room, over the slice, and a sweep that
// lists those of the selected part; then rounds of 8 bits over what is left, but for digits that all its keys share.
// Flat rows on one CTA have 5000 entries to a code, more than the list holds, equal ones all of them.  80 rows of 128256 bf16, microseconds,
// four rounds over leading bits of every key / four of the slice behind a list without room / parts: top-p of flat rows 267 / 307 / 249,
// top-k of equal rows 287 / 332 / 267, top-k with top-p and typical-p of equal rows 551 / 669 / 457.  (What it costs where the list had room:
// one row of 50272 behind typical-p 30.6 -> 32.6, 150 rows with top-p 246 -> 256; with all three 32 rows 77 -> 70, 96 rows 181 -> 180.)
template <class LoadF, class CodeF, class PartF, class KeyF, class WQ>
__device__ uint32_t select_key(Cl& c, int lo, int hi, LoadF load, CodeF code, PartF part, KeyF keyf, WQ wq, uint32_t T, bool strict, bool descending,
                               uint32_t (*hist)[HIST_WORDS], uint32_t* hsum, uint32_t* bcast, float4* xch, float* few, int* n_few, uint32_t* key_bits) {
  auto next_hist = [&]() {
    uint32_t* h = hist[c.he & 1];
    ++c.he;
    hist_clear(h);
    return h;
  };
  // put(v, digit, weight) of every entry of the slice (weight 0: does not count)
  auto add_slice = [&](auto bins, uint32_t* h, auto put) {
    for (int base = lo; base < hi; base += SAMP_THREADS * 8) {
      const int i0 = base + threadIdx.x * 8;
      uint32_t digit[8], w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (i0 < hi) {
        float v[8];
        load(i0, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) put(v[e], digit[e], w[e]);
      }
      hist_add8<decltype(bins)::value>(h, digit, w);
    }
  };
  auto list = [&](float v) {
    const int at = atomicAdd(n_few, 1);
    if (at < SAMP_FEW) few[at] = v;
  };
  constexpr std::integral_constant<int, CODES> codes{};
  uint32_t* h = next_hist();
  add_slice(codes, h, [&](float v, uint32_t& digit, uint32_t& w) {
    digit = code(v);
    w = wq(v);
  });
  hist_fold<CODES>(h);
  if (threadIdx.x == 0) {
    *n_few = 0;
    key_bits[0] = 0xffffffffu;
    key_bits[1] = 0u;
  }
  radix_round_pick<CODES>(c, h, hsum, bcast, 0u, T, strict, descending);
  const uint32_t sel = bcast[0];
  uint32_t before = bcast[1];
  for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
    if (*n_few > SAMP_FEW) break;
    float v[8];
    load(i0, v);
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (code(v[e]) == sel) list(v[e]);
  }
  h = next_hist();   // (behind its barrier the list is complete)
  const int n_code = *n_few;
  const bool code_listed = n_code <= SAMP_FEW;
  if (code_listed) {
    for (int i = threadIdx.x; i < n_code; i += SAMP_THREADS) atomicAdd(&h[(threadIdx.x & 1) * CODES + part(few[i])], wq(few[i]));
  } else {
    add_slice(codes, h, [&](float v, uint32_t& digit, uint32_t& w) {
      if (code(v) != sel) return;
      digit = part(v);
      w = wq(v);
    });
  }
  hist_fold<CODES>(h);
  if (!code_listed && threadIdx.x == 0) *n_few = 0;   // (everyone has read it)
  radix_round_pick<CODES>(c, h, hsum, bcast, before, T, strict, descending);
  const uint32_t sub = bcast[0];
  const bool some = bcast[2] != 0;
  before = bcast[1];
  uint32_t all = 0xffffffffu, any = 0u;   // key bits that every entry left has, and that any has
  auto note = [&](float v) {
    const uint32_t k = keyf(v);
    all &= k;
    any |= k;
  };
  if (code_listed) {
    for (int i = threadIdx.x; i < n_code; i += SAMP_THREADS)
      if (part(few[i]) == sub) note(few[i]);
  } else {
    for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
      float v[8];
      load(i0, v);
      const bool room = *n_few <= SAMP_FEW;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (code(v[e]) == sel && part(v[e]) == sub) {
          note(v[e]);
          if (room) list(v[e]);
        }
    }
  }
  all = __reduce_and_sync(0xffffffffu, all);
  any = __reduce_or_sync(0xffffffffu, any);
  if ((threadIdx.x & 31) == 0 && (all & ~any) == 0) {   // (of no entry: all bits and none)
    atomicAnd(&key_bits[0], all);
    atomicOr(&key_bits[1], any);
  }
  __syncthreads();
  const XchView bits = cl_publish(c, xch, Xch4{__uint_as_float(key_bits[0]), __uint_as_float(key_bits[1]), 0.f, 0.f});
  all = __reduce_and_sync(0xffffffffu, __float_as_uint(bits.mine.x));
  any = __reduce_or_sync(0xffffffffu, __float_as_uint(bits.mine.y));
  const uint32_t alike = some ? ~(all ^ any) : 0u;
  const int n = *n_few;
  uint32_t prefix = 0;
  for (int round = 0; round < 4; ++round) {
    const int shift = 24 - 8 * round;
    if (((alike >> shift) & 255) == 255) {
      prefix |= all & (255u << shift);
      continue;
    }
    auto counts = [&](uint32_t k) { return round == 0 || (k >> (shift + 8)) == (prefix >> (shift + 8)); };
    h = next_hist();
    if (n <= SAMP_FEW) {
      for (int i = threadIdx.x; i < n; i += SAMP_THREADS) {
        const uint32_t k = keyf(few[i]);
        if (part(few[i]) == sub && counts(k)) atomicAdd(&h[(threadIdx.x & 3) * 256 + ((k >> shift) & 255)], wq(few[i]));
      }
    } else {
      add_slice(std::integral_constant<int, 256>{}, h, [&](float v, uint32_t& digit, uint32_t& w) {
        const uint32_t k = keyf(v);
        digit = (k >> shift) & 255;
        if (code(v) == sel && part(v) == sub && counts(k)) w = wq(v);
      });
    }
    hist_fold<256>(h);
    radix_round_pick<256>(c, h, hsum, bcast, before, T, strict, descending);
    prefix |= bcast[0] << shift;
    before = bcast[1];
  }
  return prefix;
}
__device__ __forceinline__ uint32_t mass_target(float target) { return __float2uint_rn(fminf(fmaxf(target, 0.f), 2.f) * SAMP_FIX); }

// ---------------------------------------------------------------- Philox4x32-10
__device__ __forceinline__ uint4 philox4x32(uint4 ctr, uint2 key) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, ctr.x), lo0 = 0xD2511F53u * ctr.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, ctr.z), lo1 = 0xCD9E8D57u * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += 0x9E3779B9u;
    key.y += 0xBB67AE85u;
  }
  return ctr;
}

// ---------------------------------------------------------------- the kernel
// Grid = rows x ncl CTAs; the ncl CTAs of a row form one thread-block cluster (runtime cluster size) and each scans
// 1/ncl of the vocabulary.  Pass 1 (every row): raw max / sum-exp, and for plain greedy rows the argmax of the processed
// logits in the same sweep -- such a row costs ONE vectorised pass over its logits plus one cluster exchange.
// MASKED: some row of the launch carries a guided-decoding bitmask (a separate instantiation, so that launches without
// guided rows -- every benchmark configuration -- run exactly the code they ran before the mask existed).
template <class LT, bool MASKED>
__global__ void __launch_bounds__(SAMP_THREADS, 1)
tgis_sampler_kernel(const LT* logits, int ld, int V, const SampleRow* __restrict__ rows, uint32_t* seen_bitmap,
                    int bitmap_words, float* scratch, SampleOut* __restrict__ outs, int ncl, int cache_x, int cache_y,
                    const uint32_t* allow_bitmap) {
  // dynamic shared memory: [slice of the raw logits (cache_x)] [slice of the processed logits, fp32 (cache_y)]
  extern __shared__ __align__(16) uint8_t dyn_smem[];
  __shared__ float redf[SAMP_WARPS];
  __shared__ int redi[SAMP_WARPS];
  __shared__ uint32_t hist[2][HIST_WORDS];
  __shared__ uint32_t hsum[CODES];
  __shared__ uint32_t bcast[4];
  __shared__ uint32_t key_bits[2];
  __shared__ float4 xch[2];
  __shared__ RedBest redb[SAMP_WARPS];
  __shared__ float wmax[SAMP_WARPS];    // of the slice's raw entries, by warp
  __shared__ float cand_v[MAX_TOPN];
  __shared__ int cand_i[MAX_TOPN];
  // in turn: the entries of a selection's code, what the race is run over, what can be among the top-n, the slices' best
  __shared__ uint32_t list_words[SAMP_FEW];
  float* few = reinterpret_cast<float*>(list_words);
  float* list_v = few;
  int* list_i = reinterpret_cast<int*>(list_words + SAMP_LIST);
  __shared__ int list_n;
  STL_ENTER(6);
  griddep_launch();
  Cl cl;
  cl.ncl = ncl;
  cl.rank = ncl > 1 ? (int)cg::this_cluster().block_rank() : 0;
  cl.xe = cl.he = 0;
  const int r = blockIdx.x / ncl;
  const int crank = cl.rank;
  RowCtx<LT> c;
  c.p = rows[r];   // (written by the host before the step)
  c.V = V;
  {
    const int per = ((V + ncl - 1) / ncl + 7) / 8 * 8;
    c.lo = min(V, crank * per);
    c.hi = min(V, c.lo + per);
  }
  const int lo = c.lo, hi = c.hi;
  c.x = logits + (size_t)c.p.logits_row * ld;
  const int per_cta = ((V + ncl - 1) / ncl + 7) / 8 * 8;
  LT* xs = reinterpret_cast<LT*>(dyn_smem);
  c.xc = nullptr;  // set after pass 1 has filled it
  c.seen = (c.p.seq_slot >= 0 && c.p.rep_penalty != 1.0f) ? seen_bitmap + (size_t)c.p.seq_slot * bitmap_words : nullptr;
  c.allow = (MASKED && (c.p.flags & SAMPLE_MASKED) && c.p.seq_slot >= 0)
                ? allow_bitmap + (size_t)c.p.seq_slot * bitmap_words : nullptr;
  c.lenfac_m1 = (c.p.flags & SAMPLE_LENPEN) ? c.p.len_decay_factor : 0.f;
  c.mask_eos = c.p.n_out < c.p.min_tokens;
  c.typical = false;
  // FORCED rows (prompt logprobs): the token is given, only its raw logprob / rank / top-n are wanted
  const bool forced = (c.p.flags & SAMPLE_FORCED) != 0;
  const bool greedy = (c.p.flags & SAMPLE_GREEDY) && !forced;
  const bool want_lp = (c.p.flags & SAMPLE_LOGPROBS) != 0;
  // processed logits (sampling rows only): shared memory when the slice fits, else the global scratch row; indexed y[i]
  float* y = cache_y ? reinterpret_cast<float*>(dyn_smem + (cache_x ? (size_t)per_cta * sizeof(LT) : 0)) - lo
                     : scratch + (size_t)r * V;

  griddep_wait();
  STL_WAITED();

  // ---- pass 1: raw max / sum-exp (+ greedy argmax of the processed logits in the same sweep); the slice is staged in
  // shared memory on the way when it fits
  MaxSum ms{-INFINITY, 0.f, 0.f};
  ValIdx best{-INFINITY, -1};
  const bool do_typ = (c.p.flags & SAMPLE_TYPICAL) != 0 && !forced;
  const bool greedy_fast = greedy && !do_typ;  // argmax fused into the first sweep
  // a batch of entries at once: their maximum, then exponentials that do not wait for one another
  auto batch_max = [&](float m) {
    if (m > ms.m) ms = ms_against(ms, m);
  };
  auto consume8 = [&](float (&xs)[8], int i0) {
    float s0 = 0.f, s1 = 0.f;
    if (ms.m == -INFINITY) {   // (nothing allowed so far)
    } else if (do_typ) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = xs[e] - ms.m, p = expf(d);
        s0 += p;
        s1 += d == -INFINITY ? 0.f : d * p;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        s0 += __expf(xs[e] - ms.m);
        s1 += __expf(xs[e + 1] - ms.m);
      }
      s0 += s1;
    }
    ms.s += s0;
    if (do_typ) ms.w += s1;
    if (greedy_fast) {
      process8(c, i0, xs);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (best.i < 0 || xs[e] > best.v) best = {xs[e], i0 + e};  // ascending i: strict > keeps the lowest index
    }
  };
  constexpr int P1_UNROLL = 4;  // 16-byte loads in flight per thread (64 KB per SM)
  for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8 * P1_UNROLL) {
    float xv[P1_UNROLL][8];
#pragma unroll
    for (int u = 0; u < P1_UNROLL; ++u) {
      const int iu = i0 + u * SAMP_THREADS * 8;
      if (iu < hi) load_x8(c.x, iu, xv[u]);
    }
    float m = -INFINITY;
#pragma unroll
    for (int u = 0; u < P1_UNROLL; ++u) {
      const int iu = i0 + u * SAMP_THREADS * 8;
      if (iu < hi) {
        if (MASKED && c.allow != nullptr) {  // iu % 8 == 0: the 8 bits of this group sit in one byte of the bitmap
          const uint32_t bits = (c.allow[iu >> 5] >> (iu & 31)) & 0xffu;
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (!((bits >> e) & 1u)) xv[u][e] = -INFINITY;
        }
        if (cache_x) store_x8(xs + (iu - lo), xv[u]);
#pragma unroll
        for (int e = 0; e < 8; ++e) m = fmaxf(m, xv[u][e]);
      }
    }
    batch_max(m);
#pragma unroll
    for (int u = 0; u < P1_UNROLL; ++u) {
      const int iu = i0 + u * SAMP_THREADS * 8;
      if (iu < hi) consume8(xv[u], iu);
    }
  }
  if (cache_x) c.xc = xs;  // visible to every thread after the barriers of the reductions below
  const int n_topn = min(c.p.n_topn, MAX_TOPN);
  if (n_topn > 0) {
    float m = ms.m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;   // (read behind the barriers of the reductions)
  }
  int token;
  {
    // one exchange for all of it: {max, sum-exp, best value, best index}, or {max, sum-exp, the entropy's sum}
    const MaxSumBest t = block_maxsum_best(MaxSumBest{ms, best}, redb);
    const XchView w = cl_publish(cl, xch, Xch4{t.ms.m, t.ms.s, greedy_fast ? t.best.v : t.ms.w, __int_as_float(t.best.i)});
    const bool in = (int)(threadIdx.x & 31) < ncl;
    const MaxSumBest all = warp_maxsum_best(MaxSumBest{{in ? w.mine.x : -INFINITY, in ? w.mine.y : 0.f, in && !greedy_fast ? w.mine.z : 0.f},
                                                       {in && greedy_fast ? w.mine.z : -INFINITY, in && greedy_fast ? __float_as_int(w.mine.w) : -1}});
    ms = all.ms;
    token = all.best.i;
  }
  c.raw_max = ms.m;
  c.raw_logz = logf(ms.s);

  // ---- typical-p threshold (R8): entropy, then weighted select over s = |-lp - H| ascending
  if (do_typ) {
    c.ent = c.raw_logz - ms.w / ms.s;   // -sum p log p with log p = (x - max) - log z
    const float rm = c.raw_max, lz = c.raw_logz, ent = c.ent;
    const RowCtx<LT>& cr = c;
    auto load = [&cr](int i0, float (&v)[8]) { load_slice8(cr, i0, v); };
    auto keyf = [=](float x) {
      const float lp = (x - rm) - lz;
      return __float_as_uint(fabsf((-lp) - ent));
    };
    auto code = [=](float x) { return distance_code(fabsf((-((x - rm) - lz)) - ent)); };
    auto fine = [=](float x) { return distance_part(fabsf((-((x - rm) - lz)) - ent)); };
    auto wq = [=](float x) { return __float2uint_rn(expf((x - rm) - lz) * SAMP_FIX); };
    const uint32_t k = select_key(cl, lo, hi, load, code, fine, keyf, wq, mass_target(c.p.typical_p), false, false, hist, hsum, bcast, xch, few, &list_n, key_bits);
    c.typ_thr = __uint_as_float(k);
    c.typical = true;
  }
  if (forced) {
    token = (int)c.p.seed_lo;
  } else if (greedy) {
    if (!greedy_fast) {  // typical-p + greedy (method SAMPLE, temperature 0): argmax after the mask is known
      for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
        float x[8];
        load_slice8(c, i0, x);
        process8(c, i0, x);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (best.i < 0 || x[e] > best.v) best = {x[e], i0 + e};
      }
      best = cluster_argmax(cl, best, redf, redi, xch);
      token = best.i;
    }
  } else {
    // ---- processed logits / temperature and their maximum; kept in y for what follows, but behind typical-p alone, where few
    // entries are left, made again
    float mx = -INFINITY;
    const float temp = c.p.temperature;
    const bool use_topk = c.p.top_k > 0 && c.p.top_k < V, use_topp = c.p.top_p < 1.0f,
               keep_y = use_topk || use_topp || !c.typical || c.ent > SAMP_FLAT;
    auto scaled8 = [&](int i0, float (&v)[8]) {
      load_slice8(c, i0, v);
      process8(c, i0, v);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (v[e] != -INFINITY) v[e] = __fdiv_rn(v[e], temp);   // (-inf behind typical-p: the quotient is -inf too)
    };
    auto load_y = [=](int i0, float (&v)[8]) { load_x8(y, i0, v); };
    if (threadIdx.x == 0) list_n = 0;
    __syncthreads();
    for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
      float v[8];
      scaled8(i0, v);
      if (keep_y) store_x8(y + i0, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        mx = fmaxf(mx, v[e]);
        if (!keep_y && v[e] > -INFINITY && list_n <= SAMP_LIST) {   // what typical-p left: mostly a few (numbers, as in the sweep below)
          const int at = atomicAdd(&list_n, 1);
          if (at < SAMP_LIST) {
            list_v[at] = v[e];
            list_i[at] = i0 + e;
          }
        }
      }
    }
    mx = cluster_max(cl, mx, redf, xch);
    // ---- top-k (S6): keep y >= k-th largest value
    float lo_thr = -INFINITY;
    auto keyf = [](float v) { return f2key(v); };
    auto code = [=](float v) {   // of the distance below the maximum (no number: the maximum is infinite, or v is none)
      const float t = mx - v;
      return t == t ? CODES - 1 - distance_code(t) : CODES - 1;
    };
    auto fine = [=](float v) {
      const float t = mx - v;
      return t == t ? CODES - 1 - distance_part(t) : CODES - 1;
    };
    if (use_topk) {   // (with fewer than k entries left it is the smallest of them)
      auto wq = [](float v) { return v > -INFINITY ? 1u : 0u; };   // (numbers: a NaN's code and key are not in one order)
      lo_thr = key2f(select_key(cl, lo, hi, load_y, code, fine, keyf, wq, (uint32_t)c.p.top_k, false, true, hist, hsum, bcast, xch, few, &list_n, key_bits));
    }
    // ---- top-p (S6): drop the low-probability tail whose cumulative mass <= 1 - p
    if (use_topp) {
      float part = 0.f;
      for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
        float v[8];
        load_y(i0, v);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (v[e] >= lo_thr) part += expf(v[e] - mx);
      }
      const float z = cluster_sumf(cl, part, redf, xch);
      const float lt = lo_thr;
      auto wq = [=](float v) { return v >= lt ? __float2uint_rn(expf(v - mx) / z * SAMP_FIX) : 0u; };
      const uint32_t k = select_key(cl, lo, hi, load_y, code, fine, keyf, wq, mass_target(1.0f - c.p.top_p), true, false, hist, hsum, bcast, xch, few, &list_n, key_bits);
      lo_thr = fmaxf(lo_thr, key2f(k));
    }
    // ---- exponential race == Gumbel max over the kept set
    const uint2 key = make_uint2(c.p.seed_lo, c.p.seed_hi);
    ValIdx bs{-INFINITY, -1};
    auto race = [&](float v, int i) {
      const uint4 rnd = philox4x32(make_uint4((uint32_t)i, c.p.step, 0u, 0u), key);
      // (24 ones and a half round to 2^24: without the limit u is one there, its score infinite, and one draw of 130 over 128256 entries
      // goes to such an entry whatever its probability)
      const float u = fminf(((float)(rnd.x >> 8) + 0.5f) * (1.0f / 16777216.0f), 1.f - 1.0f / 16777216.0f);
      // to be ahead, -log u has to be below e^(v - mx - best), and it is at least 1 - u: most entries need no logarithm (the
      // margin is a thousand times the rounding of what is compared)
      if (1.f - u > fmaf(__expf((v - mx) - bs.v), 1.001f, 1e-6f)) return;
      const float score = (v - mx) - logf(-logf(u));
      if (bs.i < 0 || score > bs.v) bs = {score, i};
    };
    if (!keep_y && list_n <= SAMP_LIST) {
      if ((int)threadIdx.x < list_n) race(list_v[threadIdx.x], list_i[threadIdx.x]);
    } else {
      for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
        float v[8];
        if (keep_y) load_y(i0, v);
        else scaled8(i0, v);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (v[e] >= lo_thr && v[e] != -INFINITY) race(v[e], i0 + e);
      }
    }
    bs = cluster_argmax(cl, bs, redf, redi, xch);
    token = bs.i;
    if (token < 0) {  // everything masked (degenerate): fall back to raw argmax
      ValIdx b2{-INFINITY, -1};
      for (int i = lo + threadIdx.x; i < hi; i += SAMP_THREADS) {
        const float v = load_x(c, i);
        if (b2.i < 0 || v > b2.v) b2 = {v, i};
      }
      b2 = cluster_argmax(cl, b2, redf, redi, xch);
      token = b2.i;
    }
  }

  // ---- logprob / rank / top-n on the RAW log-softmax (S1, S8)
  // The row's top-n is contained in the union of the slices' top-n.  A slice's n-th largest entry is no smaller than the n-th
  // largest of its warps' maxima (each a different entry, known from the first sweep), so the sweep that counts the token's
  // rank also lists the entries from that bound on, a few more than n.
  float tok_lp = 0.f;
  int rank = 0, cnt = 0;
  SampleOut* o = outs + r;
  float bound = INFINITY;
  auto nth_of_wmax = [&]() {   // ... the list is empty then
    if (threadIdx.x < 32) {
      const int l = threadIdx.x;
      const float v = l < SAMP_WARPS ? wmax[l] : -INFINITY;
      int before = 0;
#pragma unroll
      for (int j = 0; j < SAMP_WARPS; ++j) {
        const float t = __shfl_sync(0xffffffffu, v, j);
        before += (t > v || (t == v && j < l)) ? 1 : 0;
      }
      if (l == 0) {
        list_n = 0;
        bcast[0] = __float_as_uint(-INFINITY);   // (maxima that are no numbers: the sweep per entry below)
      }
      __syncwarp();
      if (before == n_topn - 1 && l < SAMP_WARPS) bcast[0] = __float_as_uint(v);
    }
    __syncthreads();
    return __uint_as_float(bcast[0]);
  };
  auto list_from = [&](float x, int i) {
    if (!(x >= bound)) return;
    const int at = atomicAdd(&list_n, 1);
    if (at < SAMP_LIST) {
      list_v[at] = x;
      list_i[at] = i;
    }
  };
  if (n_topn > 0) bound = nth_of_wmax();
  // (-inf: fewer than n warps have an entry that is allowed.  A slice that the list holds is listed as a whole then: 150 greedy rows of 1024,
  // 24.6 us by a sweep per entry, 17.4 so)
  const bool listed = n_topn > 0 && (bound > -INFINITY || hi - lo <= SAMP_LIST);
  if (want_lp || listed) {
    if (want_lp) tok_lp = (load_x_any(c, token) - c.raw_max) - c.raw_logz;
    for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
      float x[8];
      load_slice8(c, i0, x);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float lp = (x[e] - c.raw_max) - c.raw_logz;
        cnt += (lp >= tok_lp) ? 1 : 0;
        if (listed) list_from(x[e], i0 + e);
      }
    }
    cnt = block_sumi(cnt, redi);
  }
  if (n_topn > 0) {   // this CTA's own n best (value desc, index asc)
    __syncthreads();
    int found = listed ? list_n : SAMP_LIST + 1;
    // Where a few warps have the largest entries (a vocabulary in order) the list is long or full: the n-th largest of the maxima of its
    // warps' worths is a closer bound.  (One row of 50272 in order, greedy with top-5: 62 us by a sweep per entry, 13 so.)
    for (int tries = 0; listed && found > 32 * n_topn && tries < 3; ++tries) {
      const bool in = (int)threadIdx.x < min(found, SAMP_LIST);
      const float v = in ? list_v[threadIdx.x] : -INFINITY, before = bound;
      const int i = in ? list_i[threadIdx.x] : -1;
      float m = v;
#pragma unroll
      for (int o2 = 16; o2 > 0; o2 >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o2));
      if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
      __syncthreads();
      bound = fmaxf(nth_of_wmax(), before);
      if (bound == before) break;   // (ties: the list stays as it is)
      if (found <= SAMP_LIST) {
        if (in) list_from(v, i);
      } else {
        for (int i0 = lo + threadIdx.x * 8; i0 < hi; i0 += SAMP_THREADS * 8) {
          float x[8];
          load_slice8(c, i0, x);
#pragma unroll
          for (int e = 0; e < 8; ++e) list_from(x[e], i0 + e);
        }
      }
      __syncthreads();
      found = list_n;
    }
    if (found >= n_topn && found <= (bound > -INFINITY ? SAMP_LIST : 32 * n_topn)) {   // (at least n where maxima made the bound)
      if ((int)threadIdx.x < found) {
        const float v = list_v[threadIdx.x];
        const int i = list_i[threadIdx.x];
        int before = 0;
        for (int j = 0; j < found; ++j) before += (list_v[j] > v || (list_v[j] == v && list_i[j] < i)) ? 1 : 0;
        if (before < n_topn) {
          cand_v[before] = v;
          cand_i[before] = i;
        }
      }
    } else {   // masked to a few tokens, or more ties than the list holds: one sweep per entry
      float prev_v = INFINITY;
      int prev_i = -1;
      for (int n = 0; n < n_topn; ++n) {
        ValIdx b{-INFINITY, -1};
        for (int i = lo + threadIdx.x; i < hi; i += SAMP_THREADS) {
          const float v = load_x(c, i);
          const bool after = (v < prev_v) || (v == prev_v && i > prev_i);
          if (after && (b.i < 0 || v > b.v)) b = {v, i};
        }
        b = block_argmax(b, redf, redi);
        prev_v = b.v;
        prev_i = b.i < 0 ? 0x7fffffff : b.i;   // (the slice has no more: nothing comes behind that)
        if (threadIdx.x == 0) {
          cand_v[n] = b.v;
          cand_i[n] = b.i;
        }
      }
    }
  }
  if (want_lp || n_topn > 0) {   // ONE exchange for the counts and the lists; the cluster's rank-0 CTA orders the <= 8 x 12 candidates
    const XchView w = cl_publish(cl, xch, Xch4{__int_as_float(cnt), 0.f, 0.f, 0.f});
    if (want_lp)
      for (int q = 0; q < ncl; ++q) rank += __float_as_int(w.get(q).a);
    const int total = ncl * n_topn;
    if (crank == 0 && n_topn > 0) {
      const int e = threadIdx.x;
      if (e < total) {
        list_v[e] = dsmem_read(cl, cand_v + e % n_topn, e / n_topn);
        list_i[e] = dsmem_read(cl, cand_i + e % n_topn, e / n_topn);
      }
      if (e < n_topn) o->topn_ids[e] = -1;   // (only numbers that do not compare leave a place empty)
      __syncthreads();
      if (e < 8 * 32 * ((total + 31) / 32)) {   // eight threads to a candidate (whole warps)
        const int at = min(e >> 3, total - 1), i = list_i[at];
        const float v = list_v[at];
        int before = 0;
        for (int j = e & 7; j < total; j += 8) {   // (an index below zero: the slice had no more)
          const float u = list_v[j];
          const int k = list_i[j];
          before += k < 0 ? (i < 0 && j < at) : (i < 0 || u > v || (u == v && k < i));
        }
#pragma unroll
        for (int k = 1; k < 8; k <<= 1) before += __shfl_xor_sync(0xffffffffu, before, k);
        if ((e & 7) == 0 && (e >> 3) < total && before < n_topn) {
          o->topn_ids[before] = i;
          o->topn_lps[before] = (v - c.raw_max) - c.raw_logz;
        }
      }
    }
  }
  if (threadIdx.x == 0 && crank == 0) {
    o->token = token;
    o->logprob = tok_lp;
    o->rank = rank;
    o->n_topn = n_topn;
    if (c.p.seq_slot >= 0 && token >= 0)
      atomicOr(&seen_bitmap[(size_t)c.p.seq_slot * bitmap_words + (token >> 5)], 1u << (token & 31));
  }
  if (ncl > 1) cg::this_cluster().sync();  // nobody exits while a peer may still read its shared memory
  STL_EXIT();
}

// Cluster size of a launch: the most CTAs per row that run in one wave, a function of the launch's shape only, so that a captured
// CUDA graph replays the same launch.  Clusters do not fill a GPU whose groups of SMs are no multiple of them: of 148 SMs, 15
// clusters of eight and 33 of four are there at a time (16 rows in two waves of eight 24 us greedy, 57 typical-p, as fours 15 and 37; 34
// rows in fours 28 and 73, in pairs 20 and 55).  Greedy rows, which have two sweeps and as many exchanges, take four where eight only cost a
// longer exchange: one row of 8192 8.5 us against 10.3, fifteen of 32768 10.0 against 10.5.  The line lies where it was drawn before the
// candidates' list had its closer bound; since then eight are ahead by themselves from 50272 on (one row 9.8 against 10.3, of 128256 11.3
// against 13.2), which 16 steps of a 12-layer model with 50272 entries do not show (4137 us with eight, 4134 with four).
int sampler_cluster_size(int n_rows, int any_complex, int vocab, int num_sms) {
  if (const char* e = getenv("TGIS_SAMPLER_CLUSTER")) {
    const int v = atoi(e);
    if (v == 1 || v == 2 || v == 4 || v == 8) return v;
  }
  if (n_rows * 8 <= num_sms - 28 && (any_complex || vocab > 160 * 1024)) return 8;
  if (n_rows * 4 <= num_sms - 16) return 4;
  return n_rows * 2 <= num_sms ? 2 : 1;
}

template <class LT, bool MASKED>
static cudaError_t sampler_launch_tm(const LT* logits, int ld, int vocab, const SampleRow* rows, int n_rows,
                                    uint32_t* seen_bitmap, int bitmap_words, float* scratch, SampleOut* out, int ncl,
                                    int any_complex, cudaStream_t stream, const uint32_t* allow_bitmap) {
  // shared-memory staging of the CTA's slice: raw logits always when they fit, the processed row too for sampling rows
  const size_t per = (size_t)(((vocab + ncl - 1) / ncl + 7) / 8 * 8);
  constexpr size_t SMEM_BUDGET = 200 * 1024;
  int cache_x = per * sizeof(LT) <= SMEM_BUDGET ? 1 : 0;
  int cache_y = (any_complex && cache_x && per * (sizeof(LT) + 4) <= SMEM_BUDGET) ? 1 : 0;
  if (const char* e = getenv("TGIS_SAMPLER_SMEM"))
    if (e[0] == '0') cache_x = cache_y = 0;
  const size_t smem = (cache_x ? per * sizeof(LT) : 0) + (cache_y ? per * 4 : 0);
  static size_t attr_bytes = 0;
  if (smem > attr_bytes) {
    cudaError_t e = cudaFuncSetAttribute(tgis_sampler_kernel<LT, MASKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BUDGET);
    if (e != cudaSuccess) return e;
    attr_bytes = SMEM_BUDGET;
  }
  if (ncl > 1)
    return launch_k_cluster(tgis_sampler_kernel<LT, MASKED>, dim3(n_rows * ncl), dim3(SAMP_THREADS), smem, stream, ncl, logits, ld,
                            vocab, rows, seen_bitmap, bitmap_words, scratch, out, ncl, cache_x, cache_y, allow_bitmap);
  return launch_k(tgis_sampler_kernel<LT, MASKED>, dim3(n_rows), dim3(SAMP_THREADS), smem, stream, logits, ld, vocab, rows,
                  seen_bitmap, bitmap_words, scratch, out, 1, cache_x, cache_y, allow_bitmap);
}

template <class LT>
static cudaError_t sampler_launch_t(const LT* logits, int ld, int vocab, const SampleRow* rows, int n_rows,
                                    uint32_t* seen_bitmap, int bitmap_words, float* scratch, SampleOut* out, int ncl,
                                    int any_complex, cudaStream_t stream, const uint32_t* allow_bitmap) {
  if (allow_bitmap != nullptr)
    return sampler_launch_tm<LT, true>(logits, ld, vocab, rows, n_rows, seen_bitmap, bitmap_words, scratch, out, ncl,
                                       any_complex, stream, allow_bitmap);
  return sampler_launch_tm<LT, false>(logits, ld, vocab, rows, n_rows, seen_bitmap, bitmap_words, scratch, out, ncl,
                                      any_complex, stream, nullptr);
}

cudaError_t sampler_launch(const void* logits, int logits_bf16, int ld, int vocab, const SampleRow* rows, int n_rows,
                           const uint32_t* seen_bitmap, int bitmap_words, float* scratch, SampleOut* out,
                           cudaStream_t stream, int any_complex, int num_sms, const uint32_t* allow_bitmap) {
  if (n_rows <= 0) return cudaSuccess;
  if (vocab % 8 != 0 || ld % 8 != 0) return cudaErrorInvalidValue;
  const int ncl = sampler_cluster_size(n_rows, any_complex, vocab, num_sms);
  if (logits_bf16)
    return sampler_launch_t(static_cast<const __nv_bfloat16*>(logits), ld, vocab, rows, n_rows,
                            const_cast<uint32_t*>(seen_bitmap), bitmap_words, scratch, out, ncl, any_complex, stream,
                            allow_bitmap);
  return sampler_launch_t(static_cast<const float*>(logits), ld, vocab, rows, n_rows, const_cast<uint32_t*>(seen_bitmap),
                          bitmap_words, scratch, out, ncl, any_complex, stream, allow_bitmap);
}

size_t sampler_scratch_floats(int vocab) { return (size_t)vocab; }

// ---------------------------------------------------------------- seen-token bitmap maintenance
// grid (8, slots)
__global__ void bitmap_clear_kernel(uint32_t* bm, int words, BitmapSlots slots) {
  griddep_launch();
  griddep_wait();
  uint32_t* row = bm + (size_t)slots.slot[blockIdx.y] * words;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) row[i] = 0u;
}
__global__ void bitmap_set_kernel(uint32_t* bm, int words, const int32_t* slots, const int32_t* tokens, int n) {
  griddep_launch();
  griddep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = slots[i], t = tokens[i];
  if (s < 0 || t < 0 || (t >> 5) >= words) return;
  atomicOr(&bm[(size_t)s * words + (t >> 5)], 1u << (t & 31));
}
cudaError_t bitmap_clear_launch(uint32_t* bitmap, int bitmap_words, const BitmapSlots& slots, cudaStream_t stream) {
  if (slots.n <= 0) return cudaSuccess;
  if (slots.n > BITMAP_SLOTS) return cudaErrorInvalidValue;
  return launch_k(bitmap_clear_kernel, dim3(8, slots.n), dim3(256), 0, stream, bitmap, bitmap_words, slots);
}
cudaError_t bitmap_set_launch(uint32_t* bitmap, int bitmap_words, const int32_t* slots, const int32_t* tokens, int n,
                              cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  return launch_k(bitmap_set_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, bitmap, bitmap_words, slots, tokens, n);
}

}  // namespace tgis
