// Mixers that carry a state from token to token: the token shift and decayed outer-product memory of RWKV-style time
// mixing, the gated matrix memory of xLSTM (mLSTM), the short convolution and selective scan of Mamba, and the per-head
// norm + gate that follows the two memories.
//
// State lives in fp32, one slot per sequence and layer (the engine's sequence slot).  A kernel reads the slot's state
// for the first token of a portion unless that token sits at position 0 -- then the state is zero, so a slot needs no
// clearing when it passes to another sequence --, walks the portion's tokens in ascending order and leaves the state
// behind the last one.  The arithmetic of a token therefore depends on the tokens before it only, never on how the
// sequence was cut into steps, on the other sequences of the batch or on the slot.  Everything that enters a recurrence
// (decays, gates, step sizes, normalisers) is evaluated in fp32 with expf / tanhf / log1pf, no fast-math forms.
//
// The scans are sequential over tokens and parallel over what is independent: channels (selective scan), heads and
// value columns (outer-product memories).  A state update is done by the thread that owns the entry, in the launch that
// is the LAST reader of the old state in its layer, so no launch reads a state another CTA of the same launch rewrites.
#include <cstdint>

#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace tgis {
namespace {

__device__ __forceinline__ void st_op(void* out, int dt, size_t i, float v) {
  if (dt == DT_BF16) reinterpret_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(out)[i] = v;
}
template <int VEC>
__device__ __forceinline__ void ld_vec(const float* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
#pragma unroll
    for (int e = 0; e < VEC; ++e) v[e] = p[e];
  }
}
template <int VEC>
__device__ __forceinline__ void st_op_vec(void* out, int dt, size_t i, const float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    if (dt == DT_BF16) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + i) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    } else {
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + i) = make_float4(v[0], v[1], v[2], v[3]);
    }
  } else {
#pragma unroll
    for (int e = 0; e < VEC; ++e) st_op(out, dt, i + e, v[e]);
  }
}
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }
__device__ __forceinline__ float logsigmoid_f(float z) { return z >= 0.f ? -log1pf(expf(-z)) : z - log1pf(expf(z)); }
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ------------------------------------------------------------------------------------------------ token shift
// VEC = 4: 16-byte loads, 8- or 16-byte stores (needs width and out_bs to be multiples of four and the pointers aligned); one piece of
// the row per thread, so that a step of a few tokens is not a chain of loads: 32 tokens x 2048 x 5 mixes 28.9 -> 3.9 us
template <int VEC>
__global__ void __launch_bounds__(128)
token_shift_mix_kernel(const float* __restrict__ x, int width, const float* __restrict__ mu, int n_mix,
                       const int32_t* __restrict__ positions, const int32_t* __restrict__ tok_slot,
                       const float* __restrict__ prev_state, void* __restrict__ out, int out_dtype, long long out_bs) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x;
  const int slot = tok_slot[t];
  const float* prev = nullptr;   // nullptr: zeros
  if (positions[t] > 0) prev = (t > 0 && tok_slot[t - 1] == slot) ? x + (size_t)(t - 1) * width : prev_state + (size_t)slot * width;
  const int i = (blockIdx.y * 128 + threadIdx.x) * VEC;
  if (i >= width) return;
  float h[VEC], d[VEC];
  ld_vec<VEC>(x + (size_t)t * width + i, h);
#pragma unroll
  for (int e = 0; e < VEC; ++e) d[e] = 0.f;
  if (prev) ld_vec<VEC>(prev + i, d);
#pragma unroll
  for (int e = 0; e < VEC; ++e) d[e] -= h[e];
#pragma unroll 5
  for (int s = 0; s < n_mix; ++s) {
    float m[VEC];
    ld_vec<VEC>(mu + (size_t)s * width + i, m);
#pragma unroll
    for (int e = 0; e < VEC; ++e) m[e] = fmaf(d[e], m[e], h[e]);
    st_op_vec<VEC>(out, out_dtype, (size_t)s * out_bs + (size_t)t * width + i, m);
  }
}

// ------------------------------------------------------------------------------------------------ short convolution
// VEC channels per thread (VEC = 4: 16-byte loads and stores; needs ld, inner and every base pointer aligned to four floats)
template <int VEC>
__global__ void __launch_bounds__(128)
short_conv_silu_kernel(const float* __restrict__ xz, int ld, int inner, const float* __restrict__ w,
                       const float* __restrict__ b, int taps, const int32_t* __restrict__ positions,
                       const int32_t* __restrict__ tok_slot, const float* __restrict__ conv_state,
                       float* __restrict__ out_f32, void* __restrict__ out_op, int out_dtype) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x, c = (blockIdx.y * 128 + threadIdx.x) * VEC;
  if (c >= inner) return;
  const int slot = tok_slot[t], p = positions[t];
  int nb = 0;  // predecessors of this token inside the batch (as far as the taps reach)
  while (nb < taps - 1 && t - nb - 1 >= 0 && tok_slot[t - nb - 1] == slot) ++nb;
  float acc[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) acc[e] = b != nullptr ? b[c + e] : 0.f;
  if (VEC == 4 && taps == 4) {   // the usual length: all of a channel's loads are on their way before the first sum (32 tokens x 4096 7.9 -> 5.1 us)
    float v[4][4], wt[4][4];
#pragma unroll
    for (int j = 3; j >= 0; --j) {
      const float* src = j <= nb ? xz + (size_t)(t - j) * ld + c : conv_state + ((size_t)slot * 3 + (3 - j + nb)) * inner + c;
      if (p - j >= 0) ld_vec<4>(src, v[j]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) ld_vec<4>(w + (size_t)(c + e) * 4, wt[e]);
#pragma unroll
    for (int j = 3; j >= 0; --j)
      if (p - j >= 0)
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[e] = fmaf(wt[e][3 - j], v[j][e], acc[e]);
    taps = 0;
  }
  for (int j = taps - 1; j >= 0; --j) {   // oldest input first
    if (p - j < 0) continue;
    const float* src = j <= nb ? xz + (size_t)(t - j) * ld + c
                               : conv_state + ((size_t)slot * (taps - 1) + (taps - 1 - j + nb)) * inner + c;
    float v[VEC];
    if (VEC == 4) {
      const float4 q = *reinterpret_cast<const float4*>(src);
      v[0] = q.x; v[1 % VEC] = q.y; v[2 % VEC] = q.z; v[3 % VEC] = q.w;
    } else {
      v[0] = *src;
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] = fmaf(w[(size_t)(c + e) * taps + (taps - 1 - j)], v[e], acc[e]);
  }
#pragma unroll
  for (int e = 0; e < VEC; ++e) acc[e] = silu_f(acc[e]);
  if (out_f32) {
    if (VEC == 4) *reinterpret_cast<float4*>(out_f32 + (size_t)t * inner + c) = make_float4(acc[0], acc[1 % VEC], acc[2 % VEC], acc[3 % VEC]);
    else out_f32[(size_t)t * inner + c] = acc[0];
  }
  if (out_op) st_op_vec<VEC>(out_op, out_dtype, (size_t)t * inner + c, acc);
}

// The same for four taps and aligned rows, eight tokens per thread: a token's three predecessors are the values just used (the batch
// holds portions one behind the other), so an input is read once and not four times.  2048 tokens x 4096 channels: 80 -> 26 us.
constexpr int CONV_RUN = 8;
__global__ void __launch_bounds__(128)
short_conv_run_kernel(const float* __restrict__ xz, int ld, int inner, const float* __restrict__ w, const float* __restrict__ b,
                      const int32_t* __restrict__ positions, const int32_t* __restrict__ tok_slot, const float* __restrict__ conv_state,
                      float* __restrict__ out_f32, void* __restrict__ out_op, int out_dtype, int T) {
  griddep_launch();
  const int t0 = blockIdx.x * CONV_RUN, c = (blockIdx.y * 128 + threadIdx.x) * 4;
  if (c >= inner) return;
  float wt[4][4], bias[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int e = 0; e < 4; ++e) ld_vec<4>(w + (size_t)(c + e) * 4, wt[e]);
  if (b != nullptr)
#pragma unroll
    for (int e = 0; e < 4; ++e) bias[e] = b[c + e];
  griddep_wait();
  int slot[CONV_RUN + 3];
  float x[CONV_RUN + 3][4];
#pragma unroll
  for (int i = 0; i < CONV_RUN + 3; ++i) {
    const int t = t0 - 3 + i;
    slot[i] = t >= 0 && t < T ? tok_slot[t] : -1;
    if (t >= 0 && t < T) ld_vec<4>(xz + (size_t)t * ld + c, x[i]);
  }
#pragma unroll
  for (int i = 0; i < CONV_RUN; ++i) {
    const int t = t0 + i;
    if (t >= T) break;
    const int p = positions[t], s = slot[i + 3];
    int nb = 0;   // predecessors of this token inside the batch
#pragma unroll
    for (int j = 1; j < 4; ++j)
      if (nb == j - 1 && slot[i + 3 - j] == s) nb = j;
    float acc[4] = {bias[0], bias[1], bias[2], bias[3]};
#pragma unroll
    for (int j = 3; j >= 0; --j) {   // oldest input first
      if (p - j < 0) continue;
      float v[4] = {x[i + 3 - j][0], x[i + 3 - j][1], x[i + 3 - j][2], x[i + 3 - j][3]};
      if (j > nb) ld_vec<4>(conv_state + ((size_t)s * 3 + (3 - j + nb)) * inner + c, v);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = fmaf(wt[e][3 - j], v[e], acc[e]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = silu_f(acc[e]);
    if (out_f32) *reinterpret_cast<float4*>(out_f32 + (size_t)t * inner + c) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    if (out_op) st_op_vec<4>(out_op, out_dtype, (size_t)t * inner + c, acc);
  }
}

// The sequence of rank `rank` by length, longest first (ties in order), of up to sixteen; of more, whose blocks fill the chip anyway, number
// `rank` (a block's look at 64 lengths costs 2 us: 32 prompts of 32 tokens 77.7 -> 74.3 us without, 64 of 5 93.7 -> 84.4).  (seqs is
// written by the host before the step.)
constexpr int ORDERED_SEQS = 16;
__device__ __forceinline__ int longest_first(const AttnSeq* __restrict__ seqs, int n_seqs, int rank, int* lens, int* pick) {
  if (n_seqs <= 1 || n_seqs > ORDERED_SEQS) return rank;
  const int tid = threadIdx.x;
  if (tid < n_seqs) lens[tid] = seqs[tid].q_len;
  __syncthreads();
  if (tid < n_seqs) {
    int before = 0;
    for (int j = 0; j < n_seqs; ++j) before += lens[j] > lens[tid] || (lens[j] == lens[tid] && j < tid);
    if (before == rank) *pick = tid;
  }
  __syncthreads();
  return *pick;
}

// ------------------------------------------------------------------------------------------------ selective scan
constexpr int SCAN_THREADS = 64, SCAN_CHUNK = 8, SCAN_REG_STATE = 16, SCAN_LPC = 4, SCAN_RPL = SCAN_REG_STATE / SCAN_LPC;
// the convolution's tail: inputs of the last taps - 1 positions (entry e: position end - (taps - 1) + e)
__device__ __forceinline__ void scan_save_conv(const SelScan& a, const AttnSeq& sq, int slot, int c) {
  const int K1 = a.taps - 1, first = sq.kv_len - sq.q_len;
  float* cs = a.conv_state + (size_t)slot * K1 * a.inner + c;
  for (int e = 0; e < K1; ++e) {   // ascending: entry e + q_len is read before it could be rewritten
    const int pp = sq.kv_len - K1 + e;
    float v = 0.f;
    if (pp >= first) v = a.xz[(size_t)(sq.q_start + pp - first) * a.ld_xz + c];
    else if (pp >= 0) v = cs[(size_t)(e + sq.q_len) * a.inner];
    cs[(size_t)e * a.inner] = v;
  }
}
// Up to SCAN_REG_STATE states: grid (sequences * ceil(inner / 16)), SCAN_LPC lanes share a channel; lane `sub` keeps states
// 4 sub .. + 3 and their decay rates in registers.  A channel's tokens follow one another, so what is bound is the number of
// instructions a token takes, and where few channels are left their latency.  What the four lanes would all do is dealt out: of a chunk's
// CHUNK tokens a lane fetches a quarter (step size, input, gate), takes their softplus, hands step size and input on by shuffle, and after
// the chunk receives its tokens' output sums (a transposing reduction: 12 shuffles for 16 tokens and 4 lanes) and gates and writes
// them.  B and C rows go through two shared-memory buffers, read four states to a load; the next chunk's step sizes are worked out
// beside this chunk's outputs, its loads a chunk before.  Whole chunks of ALL = SCAN_REG_STATE states have no branch in them, so that the
// tokens' exponentials run beside one another and only the fma of a state waits for the token before; a sequence's last chunk tests
// its tokens one by one.  Longest sequences first.  4096 channels of 16 states, microseconds without overlap: 2048 tokens in 7 prompts 306 -> 163
// (chunks of 32: 188); the length of a chunk stands at scan_chunk.
template <bool ALL, int CHUNK>
__global__ void __launch_bounds__(SCAN_THREADS)
selective_scan_reg_kernel(SelScan a, const AttnSeq* __restrict__ seqs, int n_seqs, const int32_t* __restrict__ tok_slot) {
  constexpr int TPL = CHUNK / SCAN_LPC, ROW = 2 * SCAN_REG_STATE, STAGE = CHUNK * ROW / SCAN_THREADS;
  static_assert(SCAN_LPC == 4 && SCAN_RPL == 4, "the reduction below deals a chunk's tokens to four lanes");
  __shared__ __align__(16) float BC[2][CHUNK * ROW];   // per token: B | C, zeros behind the last state
  __shared__ int lens[ORDERED_SEQS], pick;
  griddep_launch();
  constexpr int CH = SCAN_THREADS / SCAN_LPC;
  const int n_blk = (a.inner + CH - 1) / CH, N = ALL ? SCAN_REG_STATE : a.state, tid = threadIdx.x, lane = tid & 31, sub = tid % SCAN_LPC;
  const int seq = longest_first(seqs, n_seqs, blockIdx.x / n_blk, lens, &pick);
  const AttnSeq sq = seqs[seq];
  griddep_wait();
  const int c = blockIdx.x % n_blk * CH + tid / SCAN_LPC;
  const bool live = c < a.inner;
  const int slot = tok_slot[sq.q_start];
  float* Sg = a.S + ((size_t)slot * a.inner + (live ? c : 0)) * N;
  float Sr[SCAN_RPL], Ar[SCAN_RPL];
#pragma unroll
  for (int j = 0; j < SCAN_RPL; ++j) {
    const int n = sub * SCAN_RPL + j;
    Sr[j] = (live && sq.kv_len > sq.q_len && n < N) ? Sg[n] : 0.f;
    Ar[j] = (live && n < N) ? -expf(a.A_log[(size_t)c * N + n]) : 0.f;
  }
  const float dtb = live ? a.dt_b[c] : 0.f, Dc = live ? a.D[c] : 0.f;
  float p_bc[STAGE], p_dt[TPL], p_x[TPL], p_z[TPL];
  auto fetch = [&](int t0) {
    const int nt = min(CHUNK, sq.q_len - t0);
#pragma unroll
    for (int k = 0; k < STAGE; ++k) {
      const int e = tid + k * SCAN_THREADS, tt = e / ROW, which = (e % ROW) / SCAN_REG_STATE, n = e % SCAN_REG_STATE;
      p_bc[k] = tt < nt && n < N ? a.proj[(size_t)(sq.q_start + t0 + tt) * a.ld_proj + a.dt_rank + which * N + n] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
      const size_t row = (size_t)(sq.q_start + t0 + sub * TPL + i);
      const bool ok = live && sub * TPL + i < nt;
      p_dt[i] = ok ? a.dt_raw[row * a.inner + c] : 0.f;
      p_x[i] = ok ? a.x[row * a.inner + c] : 0.f;
      p_z[i] = ok ? a.xz[row * a.ld_xz + a.inner + c] : 0.f;
    }
  };
  float dt[TPL], dx[TPL], xv[TPL], zv[TPL];
  auto stage = [&](int buf) {   // what was fetched: B and C to a buffer, the tokens' step sizes
#pragma unroll
    for (int k = 0; k < STAGE; ++k) BC[buf][tid + k * SCAN_THREADS] = p_bc[k];
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
      dt[i] = softplus_f(p_dt[i] + dtb);
      xv[i] = p_x[i];
      zv[i] = p_z[i];
      dx[i] = dt[i] * xv[i];
    }
  };
  fetch(0);
  stage(0);
  if (CHUNK < sq.q_len) fetch(CHUNK);
  for (int t0 = 0, buf = 0; t0 < sq.q_len; t0 += CHUNK, buf ^= 1) {
    const int nt = min(CHUNK, sq.q_len - t0);
    __syncthreads();   // (the other buffer is written below: everyone read it before this barrier)
    float y[CHUNK];
    auto token = [&](int tt) {
      const int from = (lane & ~(SCAN_LPC - 1)) + tt / TPL;
      const float dt_t = __shfl_sync(0xffffffffu, dt[tt % TPL], from), dx_t = __shfl_sync(0xffffffffu, dx[tt % TPL], from);
      const float4 b4 = *reinterpret_cast<const float4*>(&BC[buf][tt * ROW + sub * SCAN_RPL]);
      const float4 c4 = *reinterpret_cast<const float4*>(&BC[buf][tt * ROW + SCAN_REG_STATE + sub * SCAN_RPL]);
      const float bn[4] = {b4.x, b4.y, b4.z, b4.w}, cn[4] = {c4.x, c4.y, c4.z, c4.w};
      y[tt] = 0.f;
#pragma unroll
      for (int j = 0; j < SCAN_RPL; ++j) {
        if (ALL || sub * SCAN_RPL + j < N) {
          Sr[j] = fmaf(expf(dt_t * Ar[j]), Sr[j], dx_t * bn[j]);
          y[tt] = fmaf(Sr[j], cn[j], y[tt]);
        }
      }
    };
    if (nt == CHUNK) {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) token(tt);
    } else {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) {
        y[tt] = 0.f;
        if (tt < nt) token(tt);
      }
    }
    float half[2 * TPL], out[TPL];
#pragma unroll
    for (int i = 0; i < 2 * TPL; ++i) {
      const float keep = sub & 2 ? y[2 * TPL + i] : y[i], give = sub & 2 ? y[i] : y[2 * TPL + i];
      half[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
      const float keep = sub & 1 ? half[TPL + i] : half[i], give = sub & 1 ? half[i] : half[TPL + i];
      out[i] = fmaf(Dc, xv[i], keep + __shfl_xor_sync(0xffffffffu, give, 1)) * silu_f(zv[i]);
    }
    if (t0 + CHUNK < sq.q_len) {
      stage(buf ^ 1);
      if (t0 + 2 * CHUNK < sq.q_len) fetch(t0 + 2 * CHUNK);
    }
#pragma unroll
    for (int i = 0; i < TPL; ++i)
      if (live && sub * TPL + i < nt) st_op(a.out, a.out_dtype, (size_t)(sq.q_start + t0 + sub * TPL + i) * a.inner + c, out[i]);
  }
  if (!live) return;
#pragma unroll
  for (int j = 0; j < SCAN_RPL; ++j)
    if (sub * SCAN_RPL + j < N) Sg[sub * SCAN_RPL + j] = Sr[j];
  if (sub == 0) scan_save_conv(a, sq, slot, c);
}

// Steps whose portions are single tokens: grid (sequences, ceil(inner / 64)), four lanes a channel as above and the same sums in the
// same order, but every load is requested at once (the states' lines while the kernel before still runs) instead of a chunk's staging.
// Needs SCAN_REG_STATE states and aligned rows.  32 tokens, 4096 channels: 21.5 -> 9.0 us.
__global__ void __launch_bounds__(256)
selective_step_kernel(SelScan a, const AttnSeq* __restrict__ seqs, const int32_t* __restrict__ tok_slot) {
  constexpr int N = SCAN_REG_STATE;
  griddep_launch();
  const AttnSeq sq = seqs[blockIdx.x];   // (written by the host before the step, as the slots are)
  const int slot = tok_slot[sq.q_start], sub = threadIdx.x & 3, c = blockIdx.y * 64 + (threadIdx.x >> 2);
  const bool live = c < a.inner;
  float* Sg = a.S + ((size_t)slot * a.inner + (live ? c : 0)) * N + sub * 4;
  if (live && sub == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(Sg));
  float rate[4] = {0.f, 0.f, 0.f, 0.f};
  if (live) ld_vec<4>(a.A_log + (size_t)c * N + sub * 4, rate);
#pragma unroll
  for (int j = 0; j < 4; ++j) rate[j] = -expf(rate[j]);
  const float dtb = live ? a.dt_b[c] : 0.f, Dc = live ? a.D[c] : 0.f;
  griddep_wait();
  if (!live) return;   // (a channel's four lanes leave together)
  const size_t row = (size_t)sq.q_start;
  float Sr[4] = {0.f, 0.f, 0.f, 0.f}, bn[4], cn[4];
  if (sq.kv_len > 1) ld_vec<4>(Sg, Sr);
  const float* pr = a.proj + row * a.ld_proj + a.dt_rank;
#pragma unroll
  for (int j = 0; j < 4; ++j) bn[j] = pr[sub * 4 + j], cn[j] = pr[N + sub * 4 + j];
  const float xv = a.x[row * a.inner + c], zv = a.xz[row * a.ld_xz + a.inner + c];
  const float dt = softplus_f(a.dt_raw[row * a.inner + c] + dtb), dx = dt * xv;
  // the convolution's tail: lane `sub` moves entries sub, sub + 4, ..; it reads them before the lanes that overwrite them write
  const int K1 = a.taps - 1;
  float* cs = a.conv_state + (size_t)slot * K1 * a.inner + c;
  float y = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    Sr[j] = fmaf(expf(dt * rate[j]), Sr[j], dx * bn[j]);
    y = fmaf(Sr[j], cn[j], y);
  }
  const uint32_t four = 0xfu << (threadIdx.x & 28);
  for (int e0 = 0; e0 < K1; e0 += 4) {
    const int e = e0 + sub, pp = sq.kv_len - K1 + e;
    float v = 0.f;
    if (e < K1 && pp >= 0) v = pp == sq.kv_len - 1 ? a.xz[row * a.ld_xz + c] : cs[(size_t)(e + 1) * a.inner];
    __syncwarp(four);
    if (e < K1) cs[(size_t)e * a.inner] = v;
    __syncwarp(four);
  }
  y += __shfl_xor_sync(four, y, 2);
  y += __shfl_xor_sync(four, y, 1);
  *reinterpret_cast<float4*>(Sg) = make_float4(Sr[0], Sr[1], Sr[2], Sr[3]);
  if (sub == 0) st_op(a.out, a.out_dtype, row * a.inner + c, fmaf(Dc, xv, y) * silu_f(zv));
}

// More states: one thread per channel, state in shared memory.  A chunk's B / C rows are staged in shared memory and its per-channel
// scalars (step size, input, gate) are fetched ahead of the chunk's arithmetic, so the token loop waits for memory once per chunk.
__global__ void __launch_bounds__(SCAN_THREADS)
selective_scan_kernel(SelScan a, const AttnSeq* __restrict__ seqs, const int32_t* __restrict__ tok_slot) {
  extern __shared__ float scan_smem[];
  const int N = a.state;
  float* BC = scan_smem;                                         // [SCAN_CHUNK][2 N]
  float* Ss = BC + (size_t)SCAN_CHUNK * 2 * N;                   // [N][SCAN_THREADS]
  float* As = Ss + (size_t)N * SCAN_THREADS;                     // [N][SCAN_THREADS]
  griddep_launch();
  griddep_wait();
  const AttnSeq sq = seqs[blockIdx.x];
  const int tid = threadIdx.x, c = blockIdx.y * SCAN_THREADS + tid;
  const bool live = c < a.inner;
  const int slot = tok_slot[sq.q_start];
  const int first = sq.kv_len - sq.q_len;   // position of the portion's first token
  float* Sg = a.S + ((size_t)slot * a.inner + (live ? c : 0)) * N;
  for (int n = 0; n < N; ++n) {
    Ss[n * SCAN_THREADS + tid] = (live && first > 0) ? Sg[n] : 0.f;
    As[n * SCAN_THREADS + tid] = live ? -expf(a.A_log[(size_t)c * N + n]) : 0.f;
  }
  const float dtb = live ? a.dt_b[c] : 0.f, Dc = live ? a.D[c] : 0.f;
  for (int t0 = 0; t0 < sq.q_len; t0 += SCAN_CHUNK) {
    const int nt = min(SCAN_CHUNK, sq.q_len - t0);
    __syncthreads();
    for (int i = tid; i < nt * 2 * N; i += SCAN_THREADS) {
      const int tt = i / (2 * N), j = i % (2 * N);
      BC[i] = a.proj[(size_t)(sq.q_start + t0 + tt) * a.ld_proj + a.dt_rank + j];
    }
    float dtv[SCAN_CHUNK], xv[SCAN_CHUNK], zv[SCAN_CHUNK];
#pragma unroll
    for (int tt = 0; tt < SCAN_CHUNK; ++tt) {
      const size_t row = (size_t)(sq.q_start + t0 + tt);
      const bool ok = live && tt < nt;
      dtv[tt] = ok ? a.dt_raw[row * a.inner + c] : 0.f;
      xv[tt] = ok ? a.x[row * a.inner + c] : 0.f;
      zv[tt] = ok ? a.xz[row * a.ld_xz + a.inner + c] : 0.f;
    }
    __syncthreads();
    if (!live) continue;
#pragma unroll
    for (int tt = 0; tt < SCAN_CHUNK; ++tt) {
      if (tt < nt) {
        const size_t row = (size_t)(sq.q_start + t0 + tt);
        const float dt = softplus_f(dtv[tt] + dtb);
        const float dx = dt * xv[tt];
        const float* Bt = BC + (size_t)tt * 2 * N;
        float y = 0.f;
        for (int n = 0; n < N; ++n) {
          const float sv = fmaf(expf(dt * As[n * SCAN_THREADS + tid]), Ss[n * SCAN_THREADS + tid], dx * Bt[n]);
          Ss[n * SCAN_THREADS + tid] = sv;
          y = fmaf(sv, Bt[N + n], y);
        }
        y = fmaf(Dc, xv[tt], y);
        st_op(a.out, a.out_dtype, row * a.inner + c, y * silu_f(zv[tt]));
      }
    }
  }
  if (!live) return;
  for (int n = 0; n < N; ++n) Sg[n] = Ss[n * SCAN_THREADS + tid];
  scan_save_conv(a, sq, slot, c);
}

// ------------------------------------------------------------------------------------------------ outer-product memories
// grid (sequences, heads, ceil(vdim / 32)); 256 threads = 8 row groups (warps) x 32 value columns (lanes).  Thread (g, c)
// keeps rows 4 (g + 8 j) .. + 3 of column c in registers, two to a packed pair.  The tokens' q / k / decay vectors, value columns
// and gates are staged in shared memory OS_CHUNK tokens at a time (one wait for memory per chunk).  The recurrence itself is private
// to a thread; only a token's OUTPUT sums over the row groups.  So a thread runs through the chunk's tokens without any barrier,
// leaving its partial sums per token in shared memory, and after ONE barrier warp w sums and writes the outputs of the chunk's
// tokens w, w + 8.  What is the same for all columns is not done once per thread: the gated memory's exponentials are one warp's work
// before the token loop, and its normaliser is kept a row per thread.
// Bound by instruction issue and by the latency of a token's chain (one head's tokens are worked through one after the other, and a
// prompt has only heads * vdim / 32 blocks).  Four rows to a shared-memory load and two to an fma.  This is the kernel of keys that leave
// the last row group short, and of steps whose portions are short; other prompts have outer_run_kernel.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long x, unsigned long long y) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long x, unsigned long long y, unsigned long long z) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x), "l"(y), "l"(z));
  return d;
}
constexpr int OS_GROUPS = 8, OS_COLS = 32, OS_THREADS = OS_GROUPS * OS_COLS, OS_CHUNK = 16;
// FULL: D == RPT * OS_GROUPS, every thread's rows are there (no branch in the token loop, so a token's loads go ahead of its sums).
template <int RPT, int MODE, bool FULL>
__global__ void __launch_bounds__(OS_THREADS)
outer_scan_kernel(OuterScan a, const AttnSeq* __restrict__ seqs, const int32_t* __restrict__ tok_slot) {
  extern __shared__ __align__(16) float os_smem[];
  const int D = FULL ? RPT * OS_GROUPS : a.dim, DP = (D + 3) & ~3;
  float* vec = os_smem;                                  // [OS_CHUNK][3][DP]: q | k | w (GATED: n q)
  float* vcol = vec + (size_t)OS_CHUNK * 3 * DP;         // [OS_CHUNK][OS_COLS]
  __shared__ float part[OS_CHUNK][OS_GROUPS][OS_COLS + 1];
  __shared__ float gates[OS_CHUNK][2];                   // GATED, SSD: the decay, the factor of the outer product
  __shared__ float floor_m[OS_CHUNK];                    // GATED: e^(-m) after each token
  static_assert(OS_CHUNK % OS_GROUPS == 0, "warp w writes the outputs of the chunk's tokens w, w + OS_GROUPS, ...");
  griddep_launch();
  griddep_wait();
  const AttnSeq sq = seqs[blockIdx.x];
  const int h = blockIdx.y, tid = threadIdx.x, g = tid >> 5, lane = tid & 31;
  const int hq = a.qk_heads > 0 ? h / (a.heads / a.qk_heads) : h;   // the q / k head this head reads
  const int c0 = blockIdx.z * OS_COLS, c = c0 + lane;
  const bool col_ok = c < a.vdim;
  const int slot = tok_slot[sq.q_start];
  const bool fresh = sq.kv_len - sq.q_len == 0;
  constexpr int NG = RPT / 4;          // groups of four rows
  constexpr bool OWN_DECAY = MODE == OUTER_SCAN_DECAY || MODE == OUTER_SCAN_HGRN || MODE == OUTER_SCAN_GLA;   // a decay per row
  auto row_of = [&](int j) { return 4 * (g + (j >> 2) * OS_GROUPS) + (j & 3); };
  unsigned long long S[2 * NG];
  float* Sg = a.S + (((size_t)slot * a.heads + h) * D) * a.vdim + (col_ok ? c : 0);
#pragma unroll
  for (int j = 0; j < RPT; j += 2) {
    const int i = row_of(j);
    const float s0 = (!fresh && col_ok && i < D) ? Sg[(size_t)i * a.vdim] : 0.f;
    const float s1 = (!fresh && col_ok && i + 1 < D) ? Sg[(size_t)(i + 1) * a.vdim] : 0.f;
    S[j / 2] = pack2(s0, s1);
  }
  unsigned long long u_r[2 * NG];      // DECAY: the bonus u of this thread's rows
  float n_row = 0.f, m_run = 0.f;      // GATED: the normaliser's row tid; the running maximum (warp 0)
  const float ssd_rate = MODE == OUTER_SCAN_SSD ? -expf(a.A_log[h]) : 0.f, ssd_skip = MODE == OUTER_SCAN_SSD ? a.D[h] : 0.f;
  const float fixed_decay = (MODE == OUTER_SCAN_LIGHTNING || MODE == OUTER_SCAN_RETENTION) ? a.decay[h] : 0.f;
  if (MODE == OUTER_SCAN_DECAY) {
#pragma unroll
    for (int j = 0; j < RPT; j += 2) {
      const int i = row_of(j);
      u_r[j / 2] = pack2(i < D ? a.u[(size_t)h * D + i] : 0.f, i + 1 < D ? a.u[(size_t)h * D + i + 1] : 0.f);
    }
  }
  if (MODE == OUTER_SCAN_GATED && !fresh) {
    n_row = tid < D ? a.n[((size_t)slot * a.heads + h) * D + tid] : 0.f;
    m_run = a.m[(size_t)slot * a.heads + h];
  }
  // A chunk's raw values travel global memory -> registers -> shared memory: thread (tt = tid / 16, l = tid % 16) stages entries
  // l, l + 16, ... of token tt's vectors and two of its value columns, all loads of a chunk are issued back to back, and the
  // loads of chunk n + 1 are issued before the token loop of chunk n.
  constexpr int EPT = RPT / 2, TPT = OS_THREADS / OS_CHUNK;
  static_assert(TPT == 16 && OS_CHUNK * OS_COLS == 2 * OS_THREADS, "staging map");
  const int st_tt = tid / TPT, st_l = tid % TPT;
  float pq[EPT], pk[EPT], pd[EPT], pw[EPT], pv[2], pg0 = 0.f, pg1 = 0.f;
#pragma unroll
  for (int e = 0; e < EPT; ++e) pw[e] = OWN_DECAY && st_l + e * TPT < D ? a.w0[(size_t)h * D + st_l + e * TPT] : 0.f;
  auto fetch = [&](int t0) {
    const int nt = min(OS_CHUNK, sq.q_len - t0);
    const bool tok = st_tt < nt;
    const size_t row = (size_t)(sq.q_start + t0 + (tok ? st_tt : 0));
    const float* qr = a.q + row * a.ldq + (size_t)hq * D;
    const float* kr = MODE == OUTER_SCAN_HGRN ? nullptr : a.k + row * a.ldk + (size_t)hq * D;
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const int i = st_l + e * TPT;
      const bool in = tok && i < D;
      pq[e] = in ? qr[i] : 0.f;
      pk[e] = in ? (MODE == OUTER_SCAN_HGRN ? a.u[(size_t)h * D + i] : kr[i]) : 0.f;   // HGRN: the gate's lower bound
      if (OWN_DECAY) pd[e] = in ? a.decay_raw[row * a.ldd + (size_t)h * D + i] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int col = c0 + 2 * st_l + e;
      pv[e] = (tok && col < a.vdim) ? a.v[row * a.ldv + (size_t)h * a.vdim + col] : 0.f;
    }
    if (tid < nt) {
      const size_t grow = (size_t)(sq.q_start + t0 + tid);
      if (MODE == OUTER_SCAN_GATED) { pg0 = a.ig[grow * a.ldg + h]; pg1 = a.fg[grow * a.ldg + h]; }
      if (MODE == OUTER_SCAN_SSD) pg0 = a.step_raw[grow * a.lds + h];
    }
  };
  fetch(0);
  for (int t0 = 0; t0 < sq.q_len; t0 += OS_CHUNK) {
    const int nt = min(OS_CHUNK, sq.q_len - t0);
    __syncthreads();   // the previous chunk's vectors and partial sums are consumed
    if (st_tt < nt) {
      float* v3 = vec + (size_t)st_tt * 3 * DP;
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const int i = st_l + e * TPT;
        if (i < D) {
          if (MODE == OUTER_SCAN_HGRN) {   // q = silu(.), f = l + (1 - l) sigmoid(.), and what is written: 1 - f
            v3[i] = silu_f(pq[e]) * a.q_scale;
            const float dl = pd[e] + pw[e];
            v3[DP + i] = (1.f - pk[e]) * sigmoid_f(-dl);                 // 1 - f without the cancellation near f = 1
            v3[2 * DP + i] = pk[e] + (1.f - pk[e]) * sigmoid_f(dl);
          } else if (MODE == OUTER_SCAN_LIGHTNING) {
            v3[i] = silu_f(pq[e]) * a.q_scale;
            v3[DP + i] = silu_f(pk[e]);
          } else {
            v3[i] = pq[e] * a.q_scale;
            v3[DP + i] = pk[e];
            if (MODE == OUTER_SCAN_DECAY) v3[2 * DP + i] = expf(-expf(pd[e] + pw[e]));
            if (MODE == OUTER_SCAN_GLA) v3[2 * DP + i] = expf(logsigmoid_f(pd[e] + pw[e]) * a.inv_tau);
          }
        }
      }
    }
    vcol[st_tt * OS_COLS + 2 * st_l] = MODE == OUTER_SCAN_LIGHTNING ? silu_f(pv[0]) : pv[0];
    vcol[st_tt * OS_COLS + 2 * st_l + 1] = MODE == OUTER_SCAN_LIGHTNING ? silu_f(pv[1]) : pv[1];
    if (MODE == OUTER_SCAN_GATED && tid < 32) {   // lane t: token t's gates, and the maximum that runs through them
      float ig = 0.f, fg = 0.f, m_before = 0.f, m_after = 0.f;
      if (lane < nt) {
        ig = a.gate_cap * tanhf((pg0 + a.ig_b[h]) / a.gate_cap);
        fg = logsigmoid_f(a.gate_cap * tanhf((pg1 + a.fg_b[h]) / a.gate_cap));
      }
#pragma unroll
      for (int t = 0; t < OS_CHUNK; ++t) {
        const float it = __shfl_sync(0xffffffffu, ig, t), ft = __shfl_sync(0xffffffffu, fg, t);
        if (t < nt) {
          const float m_new = fmaxf(ft + m_run, it);
          if (lane == t) m_before = m_run, m_after = m_new;
          m_run = m_new;
        }
      }
      if (lane < nt) {
        gates[lane][0] = expf(fg + m_before - m_after);
        gates[lane][1] = expf(ig - m_after);
        floor_m[lane] = expf(-m_after);
      }
    }
    if (MODE == OUTER_SCAN_SSD && tid < nt) {   // the token's step size and the decay it gives
      const float dt = softplus_f(pg0 + a.step_b[h]);
      gates[tid][0] = expf(ssd_rate * dt);
      gates[tid][1] = dt;
    }
    __syncthreads();
    if (t0 + OS_CHUNK < sq.q_len) fetch(t0 + OS_CHUNK);   // lands while this chunk's tokens are worked through
    if (MODE == OUTER_SCAN_GATED && tid < D) {
      float nk[OS_CHUNK];   // (tokens behind the last one hold what the chunk before left: read, not used)
#pragma unroll
      for (int tt = 0; tt < OS_CHUNK; ++tt) nk[tt] = gates[tt][1] * vec[(size_t)tt * 3 * DP + DP + tid];
#pragma unroll
      for (int tt = 0; tt < OS_CHUNK; ++tt) {
        if (tt < nt) {
          float* v3 = vec + (size_t)tt * 3 * DP;
          n_row = fmaf(gates[tt][0], n_row, nk[tt]);
          v3[2 * DP + tid] = n_row * v3[tid];
        }
      }
    }
#pragma unroll (RPT <= 16 ? 2 : 1)
    for (int tt = 0; tt < nt; ++tt) {
      const float* v3 = vec + (size_t)tt * 3 * DP;
      float vc = vcol[tt * OS_COLS + lane], wd = fixed_decay;
      if (MODE == OUTER_SCAN_SSD || MODE == OUTER_SCAN_GATED) vc *= gates[tt][1], wd = gates[tt][0];
      const unsigned long long vc2 = pack2(vc, vc), wd2 = pack2(wd, wd);
      unsigned long long o01 = 0, o23 = 0;   // two packed zeros
      auto step = [&](unsigned long long& s, unsigned long long& o, unsigned long long q2, unsigned long long k2, unsigned long long w2,
                      unsigned long long u2) {
        const unsigned long long kv = mul2(k2, vc2);
        if (MODE == OUTER_SCAN_DECAY) {
          o = fma2(q2, fma2(u2, kv, s), o);
          s = fma2(w2, s, kv);
        } else {
          s = fma2(w2, s, kv);
          o = fma2(q2, s, o);
        }
      };
#pragma unroll
      for (int j = 0; j < NG; ++j) {
        const int i = 4 * (g + j * OS_GROUPS);
        if (FULL || i + 4 <= D) {
          const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(v3 + i), k4 = *reinterpret_cast<const ulonglong2*>(v3 + DP + i);
          ulonglong2 w4 = make_ulonglong2(wd2, wd2);
          if (OWN_DECAY) w4 = *reinterpret_cast<const ulonglong2*>(v3 + 2 * DP + i);
          step(S[2 * j], o01, q4.x, k4.x, w4.x, u_r[2 * j]);
          step(S[2 * j + 1], o23, q4.y, k4.y, w4.y, u_r[2 * j + 1]);
        } else if (i < D) {   // the last one to three rows: what lies behind them takes no part, whatever the values are
          auto tail = [&](unsigned long long& s, unsigned long long& o, unsigned long long u, int at) {
            if (at >= D) return;
            const float2 s_was = unpack2(s), o_was = unpack2(o);
            const bool two = at + 1 < D;
            const float w0 = OWN_DECAY ? v3[2 * DP + at] : wd, w1 = OWN_DECAY && two ? v3[2 * DP + at + 1] : wd;
            step(s, o, pack2(v3[at], two ? v3[at + 1] : 0.f), pack2(v3[DP + at], two ? v3[DP + at + 1] : 0.f), pack2(w0, w1), u);
            if (!two) s = pack2(unpack2(s).x, s_was.y), o = pack2(unpack2(o).x, o_was.y);
          };
          tail(S[2 * j], o01, u_r[2 * j], i);
          tail(S[2 * j + 1], o23, u_r[2 * j + 1], i + 2);
        }
      }
      const float2 oa = unpack2(o01), ob = unpack2(o23);
      part[tt][g][lane] = (oa.x + oa.y) + (ob.x + ob.y);
    }
    __syncthreads();   // the chunk's partial sums are complete
    for (int tt = g; tt < nt; tt += OS_GROUPS) {   // this warp's tokens of the chunk
      float sum = 0.f;
#pragma unroll
      for (int r = 0; r < OS_GROUPS; ++r) sum += part[tt][r][lane];
      if (MODE == OUTER_SCAN_GATED) {
        float d = 0.f;
        for (int i = lane; i < D; i += 32) d += vec[(size_t)tt * 3 * DP + 2 * DP + i];
        d = warp_sum_f(d);
        sum = sum / (fmaxf(fabsf(d), floor_m[tt]) + 1e-6f);
      }
      if (MODE == OUTER_SCAN_SSD) sum = fmaf(ssd_skip, vcol[tt * OS_COLS + lane], sum);
      if (col_ok) a.out[(size_t)(sq.q_start + t0 + tt) * a.ldo + (size_t)h * a.vdim + c] = sum;
    }
  }
  // ---- leave the state behind the portion's last token
  if (col_ok) {
#pragma unroll
    for (int j = 0; j < RPT; j += 2) {
      const int i = row_of(j);
      const float2 s = unpack2(S[j / 2]);
      if (i < D) Sg[(size_t)i * a.vdim] = s.x;
      if (i + 1 < D) Sg[(size_t)(i + 1) * a.vdim] = s.y;
    }
  }
  // The normaliser and the running maximum belong to all column blocks of the head, each of which started from them.  More blocks
  // than the chip holds at once do not start together, so only the one that gets here last may overwrite them.
  if (MODE == OUTER_SCAN_GATED) {
    __shared__ int last_block;
    __syncthreads();   // every thread's row of n and m are read
    if (tid == 0) {
      int32_t* done = a.done + (size_t)slot * a.heads + h;
      last_block = gridDim.z == 1 || atomicAdd(done, 1) == (int)gridDim.z - 1;
      if (last_block && gridDim.z > 1) *done = 0;
    }
    __syncthreads();
    if (last_block) {
      if (tid < D) a.n[((size_t)slot * a.heads + h) * D + tid] = n_row;
      if (tid == 0) a.m[(size_t)slot * a.heads + h] = m_run;
    }
  }
  if (blockIdx.z == 0) {
    if (a.x_last != nullptr && h == 0) {
      const float* src = a.x + (size_t)(sq.q_start + sq.q_len - 1) * a.width;
      for (int i = tid; i < a.width; i += OS_THREADS) a.x_last[(size_t)slot * a.width + i] = src[i];
    }
  }
}

// Portions of several tokens whose keys fill the row groups (dim = 8 RPT): the sums of the kernel above in the same order, bit for bit.
// There a thread has one column, so that two 16-byte loads feed six packed operations, and everyone waits at a chunk's barriers while a
// few lanes take exponentials.  Here a row thread has two neighbouring columns of its group's rows, and what is not the recurrence is
// others' work: four warps fetch and stage the tokens' vectors, four rows to an instruction (the first of them also runs the gates, 32
// tokens at a time and a block of them ahead), two sum and write the outputs.  Rows, writers and stagers hand a chunk's buffer round by
// a named barrier each.  Longest sequences first: a piece's tokens follow one another, so the launch ends with the longest.
// Bound by instruction issue, of which the rows' packed multiply-adds are a third.  2048 tokens in 7 prompts (838 the longest), microseconds
// without overlap, before -> here: gated, 8 heads of 128 x 256, 302 -> 136; decayed, 32 heads of 64 x 64, 234 -> 106; 32 prompts of 64 tokens 137 ->
// 119 and 92 -> 90.  Slower: four columns a thread or 64 a piece (gated 184 to 194), chunks of eight tokens in a ring of four (154), one helping
// group for all of it (174), vectors staged number by number (155).  Rows that 16-byte loads do not reach come in four loads each: gated 165
// (311 in the kernel above while it knew full row groups, 481 since it tests every one), decayed 112 (222, 243), 256-row keys 229 (289, 587).
template <int MODE>
constexpr bool OS_OWN_DECAY = MODE == OUTER_SCAN_DECAY || MODE == OUTER_SCAN_HGRN || MODE == OUTER_SCAN_GLA;   // a decay per row
template <int MODE>
constexpr int OS_VECS = OS_OWN_DECAY<MODE> || MODE == OUTER_SCAN_GATED ? 3 : 2;   // q | k | w (GATED: n q)
constexpr int RUN_CHUNK = 16, RUN_RING = 2;
constexpr int RUN_ROWS = OS_THREADS / 2, RUN_STAGE = 128, RUN_WRITE = 64, RUN_THREADS = RUN_ROWS + RUN_STAGE + RUN_WRITE;
template <int RPT, int MODE>
constexpr size_t RUN_SMEM = (size_t)RUN_RING * RUN_CHUNK * (OS_VECS<MODE> * RPT * OS_GROUPS + (MODE == OUTER_SCAN_SSD ? 2 : 1) * OS_COLS + OS_GROUPS * OS_COLS) * sizeof(float);
// barrier ID + i, i < RUN_RING (ids as constants: one in a register would reserve all sixteen)
template <int ID>
__device__ __forceinline__ void bar_sync_at(int i, int threads) {
  if (i == 0) asm volatile("bar.sync %0, %1;\n" ::"n"(ID), "r"(threads) : "memory");
  else asm volatile("bar.sync %0, %1;\n" ::"n"(ID + 1), "r"(threads) : "memory");
}
template <int ID>
__device__ __forceinline__ void bar_arrive_at(int i, int threads) {
  if (i == 0) asm volatile("bar.arrive %0, %1;\n" ::"n"(ID), "r"(threads) : "memory");
  else asm volatile("bar.arrive %0, %1;\n" ::"n"(ID + 1), "r"(threads) : "memory");
}

template <int RPT, int MODE, bool VEC16>   // VEC16: q, k and decay rows begin on 16 bytes
__global__ void __launch_bounds__(RUN_THREADS, RPT <= 16 ? 2 : 1)
outer_run_kernel(OuterScan a, const AttnSeq* __restrict__ seqs, int n_seqs, const int32_t* __restrict__ tok_slot) {
  constexpr int D = RPT * OS_GROUPS, NV = OS_VECS<MODE>, C = RUN_CHUNK, RING = RUN_RING, CT = 2, NG = RPT / 4, UNROLL = RPT <= 16 ? 2 : 1;
  constexpr int FULL = 1, DONE = FULL + RUN_RING, EMPTY = DONE + RUN_RING, STAGED = EMPTY + RUN_RING;   // barriers: stagers -> rows -> writers -> stagers
  static_assert(RING == 2 && 32 % C == 0, "barriers; blocks of gates");
  constexpr bool GATES = MODE == OUTER_SCAN_GATED || MODE == OUTER_SCAN_SSD;
  extern __shared__ __align__(16) float os_smem[];
  float* vec = os_smem;                              // [RING][C][NV][D]
  float* vcol = vec + RING * C * NV * D;         // [RING][C][OS_COLS], times the token's factor
  float* part = vcol + RING * C * OS_COLS;       // [RING][C][OS_GROUPS][OS_COLS]
  float* vraw = part + RING * C * OS_GROUPS * OS_COLS;   // SSD: [RING][C][OS_COLS]
  __shared__ float gates[3][32][2], floor_m[3][32];  // as above, of three blocks of 32 tokens: one is made while chunks of the two before it are in the ring
  __shared__ int lens[ORDERED_SEQS], pick, last_block;
  griddep_launch();
  const int tid = threadIdx.x, nz = (a.vdim + OS_COLS - 1) / OS_COLS, piece = blockIdx.x % (a.heads * nz);
  const int seq = longest_first(seqs, n_seqs, blockIdx.x / (a.heads * nz), lens, &pick);
  const AttnSeq sq = seqs[seq];
  const int h = piece / nz, zb = piece % nz, c0 = zb * OS_COLS;
  const int hq = a.qk_heads > 0 ? h / (a.heads / a.qk_heads) : h;   // the q / k head this head reads
  const int n_chunks = (sq.q_len + C - 1) / C;
  griddep_wait();
  const int slot = tok_slot[sq.q_start];
  const bool fresh = sq.kv_len - sq.q_len == 0;
  auto block_of = [](int n) { return n * C / 32 % 3; };   // gates of chunk n: row block_of(n), from n * C % 32 on
  constexpr int EPT = C * D / 4 / RUN_STAGE, TSTEP = RUN_STAGE * 4 / D, VPT = C * OS_COLS / RUN_STAGE, NR = (D + RUN_STAGE - 1) / RUN_STAGE;
  const int ht = tid - RUN_ROWS, lane = tid & 31;
  float n_row[NR], m_run = 0.f;                      // GATED, stagers: the normaliser's rows ht, ht + 128; the running maximum (first warp)
#pragma unroll
  for (int r = 0; r < NR; ++r) n_row[r] = 0.f;
  if (tid < RUN_ROWS) {
    // ===================== the recurrence: two columns of the rows 4 (g + 8 j) .. + 3 =====================
    constexpr int LPG = OS_COLS / CT;                   // lanes of a row group
    const int g = tid / LPG, c = c0 + (tid % LPG) * CT;
    auto row_of = [&](int j) { return 4 * (g + (j >> 2) * OS_GROUPS) + (j & 3); };
    float* Sg = a.S + (((size_t)slot * a.heads + h) * D) * a.vdim + c;
    unsigned long long S[CT][2 * NG];
#pragma unroll
    for (int j = 0; j < RPT; j += 2)
#pragma unroll
      for (int e = 0; e < CT; ++e) {
        const bool in = !fresh && c + e < a.vdim;
        const float s0 = in ? Sg[(size_t)row_of(j) * a.vdim + e] : 0.f, s1 = in ? Sg[(size_t)row_of(j + 1) * a.vdim + e] : 0.f;
        S[e][j / 2] = pack2(s0, s1);
      }
    unsigned long long u_r[2 * NG];                  // DECAY: the bonus u of this thread's rows
    if (MODE == OUTER_SCAN_DECAY) {
#pragma unroll
      for (int j = 0; j < RPT; j += 2) u_r[j / 2] = pack2(a.u[(size_t)h * D + row_of(j)], a.u[(size_t)h * D + row_of(j) + 1]);
    }
    const float fixed_decay = (MODE == OUTER_SCAN_LIGHTNING || MODE == OUTER_SCAN_RETENTION) ? a.decay[h] : 0.f;
    for (int n = 0; n < n_chunks; ++n) {
      const int buf = n % RING;
      const float* v3 = vec + (size_t)buf * C * NV * D + 4 * g;
      const float* vc_from = vcol + buf * C * OS_COLS + (tid % LPG) * CT;
      const float* gate = &gates[block_of(n)][n * C % 32][0];
      float* to = part + ((size_t)buf * C * OS_GROUPS + g) * OS_COLS + (tid % LPG) * CT;
      auto token = [&](int tt) {
        unsigned long long vc2[CT], o01[CT], o23[CT];
        const float2 vc = *reinterpret_cast<const float2*>(vc_from + tt * OS_COLS);
        const float wd = GATES ? gate[2 * tt] : fixed_decay;
        const unsigned long long wd2 = pack2(wd, wd);
        vc2[0] = pack2(vc.x, vc.x);
        vc2[1] = pack2(vc.y, vc.y);
#pragma unroll
        for (int e = 0; e < CT; ++e) o01[e] = 0, o23[e] = 0;   // packed zeros
        auto step = [&](unsigned long long& s, unsigned long long& o, unsigned long long q2, unsigned long long k2, unsigned long long w2,
                        unsigned long long u2, unsigned long long v2) {
          const unsigned long long kv = mul2(k2, v2);
          if (MODE == OUTER_SCAN_DECAY) {
            o = fma2(q2, fma2(u2, kv, s), o);
            s = fma2(w2, s, kv);
          } else {
            s = fma2(w2, s, kv);
            o = fma2(q2, s, o);
          }
        };
        const float* vt = v3 + tt * NV * D;
#pragma unroll
        for (int j = 0; j < NG; ++j) {
          const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(vt + 4 * j * OS_GROUPS), k4 = *reinterpret_cast<const ulonglong2*>(vt + D + 4 * j * OS_GROUPS);
          ulonglong2 w4 = make_ulonglong2(wd2, wd2);
          if (OS_OWN_DECAY<MODE>) w4 = *reinterpret_cast<const ulonglong2*>(vt + 2 * D + 4 * j * OS_GROUPS);
#pragma unroll
          for (int e = 0; e < CT; ++e) {
            step(S[e][2 * j], o01[e], q4.x, k4.x, w4.x, u_r[2 * j], vc2[e]);
            step(S[e][2 * j + 1], o23[e], q4.y, k4.y, w4.y, u_r[2 * j + 1], vc2[e]);
          }
        }
        float sum[CT];
#pragma unroll
        for (int e = 0; e < CT; ++e) {
          const float2 oa = unpack2(o01[e]), ob = unpack2(o23[e]);
          sum[e] = (oa.x + oa.y) + (ob.x + ob.y);
        }
        *reinterpret_cast<float2*>(to + tt * OS_GROUPS * OS_COLS) = make_float2(sum[0], sum[1]);
      };
      bar_sync_at<FULL>(buf, RUN_ROWS + RUN_STAGE);
      const int nt = min(C, sq.q_len - n * C);
      if (nt == C) {
#pragma unroll UNROLL
        for (int tt = 0; tt < C; ++tt) token(tt);
      } else {
#pragma unroll 1
        for (int tt = 0; tt < nt; ++tt) token(tt);
      }
      bar_arrive_at<DONE>(buf, RUN_ROWS + RUN_WRITE);
    }
    // ---- leave the state behind the portion's last token
#pragma unroll
    for (int j = 0; j < RPT; j += 2)
#pragma unroll
      for (int e = 0; e < CT; ++e)
        if (c + e < a.vdim) {
          const float2 s = unpack2(S[e][j / 2]);
          Sg[(size_t)row_of(j) * a.vdim + e] = s.x;
          Sg[(size_t)row_of(j + 1) * a.vdim + e] = s.y;
        }
  } else if (ht < RUN_STAGE) {
    // ===================== gates, vectors, normaliser =====================
    const float ssd_rate = MODE == OUTER_SCAN_SSD ? -expf(a.A_log[h]) : 0.f;
    // a thread stages rows row4 .. + 3 of the tokens tok, tok + TSTEP, ... of a chunk
    const int row4 = ht * 4 % D, tok = ht * 4 / D;
    float4 pq[EPT], pk[EPT], pd[EPT];
    float pv[VPT], w0[4], low[4], pg0 = 0.f, pg1 = 0.f;   // (HGRN: low is the gate's lower bound)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w0[k] = OS_OWN_DECAY<MODE> ? a.w0[(size_t)h * D + row4 + k] : 0.f;
      low[k] = MODE == OUTER_SCAN_HGRN ? a.u[(size_t)h * D + row4 + k] : 0.f;
    }
    if (MODE == OUTER_SCAN_GATED && !fresh) {
      m_run = a.m[(size_t)slot * a.heads + h];
#pragma unroll
      for (int r = 0; r < NR; ++r)
        if (ht + r * RUN_STAGE < D) n_row[r] = a.n[((size_t)slot * a.heads + h) * D + ht + r * RUN_STAGE];
    }
    const float* q_at = a.q + (size_t)(sq.q_start + tok) * a.ldq + (size_t)hq * D + row4;
    const float* k_at = MODE == OUTER_SCAN_HGRN ? nullptr : a.k + (size_t)(sq.q_start + tok) * a.ldk + (size_t)hq * D + row4;
    const float* d_at = OS_OWN_DECAY<MODE> ? a.decay_raw + (size_t)(sq.q_start + tok) * a.ldd + (size_t)h * D + row4 : nullptr;
    const float* v_at = a.v + (size_t)(sq.q_start + ht / OS_COLS) * a.ldv + (size_t)h * a.vdim + c0 + lane;
    const bool v_in = c0 + lane < a.vdim;
    auto fetch = [&](int n) {
      const int nt = min(C, sq.q_len - n * C);
      auto row = [&](const float* p, bool in) {
        if (!in) return make_float4(0.f, 0.f, 0.f, 0.f);
        return VEC16 ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
      };
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const bool in = tok + e * TSTEP < nt;
        pq[e] = row(q_at + (size_t)(e * TSTEP) * a.ldq, in);
        if (MODE != OUTER_SCAN_HGRN) pk[e] = row(k_at + (size_t)(e * TSTEP) * a.ldk, in);
        if (OS_OWN_DECAY<MODE>) pd[e] = row(d_at + (size_t)(e * TSTEP) * a.ldd, in);
      }
#pragma unroll
      for (int e = 0; e < VPT; ++e) pv[e] = v_in && ht / OS_COLS + 4 * e < nt ? v_at[(size_t)(4 * e) * a.ldv] : 0.f;
      q_at += (size_t)C * a.ldq;
      if (MODE != OUTER_SCAN_HGRN) k_at += (size_t)C * a.ldk;
      if (OS_OWN_DECAY<MODE>) d_at += (size_t)C * a.ldd;
      v_at += (size_t)C * a.ldv;
    };
    auto fetch_gates = [&](int blk) {                // first warp, lane: token 32 blk + lane
      const int t = blk * 32 + lane;
      if (t >= sq.q_len) return;
      const size_t row = (size_t)(sq.q_start + t);
      if (MODE == OUTER_SCAN_GATED) { pg0 = a.ig[row * a.ldg + h]; pg1 = a.fg[row * a.ldg + h]; }
      if (MODE == OUTER_SCAN_SSD) pg0 = a.step_raw[row * a.lds + h];
    };
    auto take_gates = [&](int blk) {                 // ... the token's gates, and the maximum that runs through them
      const int nt = min(32, sq.q_len - blk * 32), at = blk % 3;
      if (MODE == OUTER_SCAN_GATED) {
        float ig = 0.f, fg = 0.f, m_before = 0.f, m_after = 0.f;
        if (lane < nt) {
          ig = a.gate_cap * tanhf((pg0 + a.ig_b[h]) / a.gate_cap);
          fg = logsigmoid_f(a.gate_cap * tanhf((pg1 + a.fg_b[h]) / a.gate_cap));
        }
#pragma unroll
        for (int t = 0; t < 32; ++t) {
          const float it = __shfl_sync(0xffffffffu, ig, t), ft = __shfl_sync(0xffffffffu, fg, t);
          if (t < nt) {
            const float m_new = fmaxf(ft + m_run, it);
            if (lane == t) m_before = m_run, m_after = m_new;
            m_run = m_new;
          }
        }
        if (lane < nt) {
          gates[at][lane][0] = expf(fg + m_before - m_after);
          gates[at][lane][1] = expf(ig - m_after);
          floor_m[at][lane] = expf(-m_after);
        }
      }
      if (MODE == OUTER_SCAN_SSD && lane < nt) {     // the token's step size and the decay it gives
        const float dt = softplus_f(pg0 + a.step_b[h]);
        gates[at][lane][0] = expf(ssd_rate * dt);
        gates[at][lane][1] = dt;
      }
    };
    auto stage = [&](int n) {
      const int buf = n % RING, nt = min(C, sq.q_len - n * C);
      const float* gate = &gates[block_of(n)][n * C % 32][0];
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        float* v3 = vec + ((size_t)(buf * C + tok + e * TSTEP) * NV) * D + row4;
        float q[4] = {pq[e].x, pq[e].y, pq[e].z, pq[e].w}, k[4] = {pk[e].x, pk[e].y, pk[e].z, pk[e].w}, w[4] = {pd[e].x, pd[e].y, pd[e].z, pd[e].w};
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          if (MODE == OUTER_SCAN_HGRN) {             // q = silu(.), f = l + (1 - l) sigmoid(.), and what is written: 1 - f
            const float dl = w[x] + w0[x];
            k[x] = (1.f - low[x]) * sigmoid_f(-dl);  // 1 - f without the cancellation near f = 1
            w[x] = low[x] + (1.f - low[x]) * sigmoid_f(dl);
          }
          if (MODE == OUTER_SCAN_LIGHTNING) k[x] = silu_f(k[x]);
          if (MODE == OUTER_SCAN_DECAY) w[x] = expf(-expf(w[x] + w0[x]));
          if (MODE == OUTER_SCAN_GLA) w[x] = expf(logsigmoid_f(w[x] + w0[x]) * a.inv_tau);
          q[x] = (MODE == OUTER_SCAN_HGRN || MODE == OUTER_SCAN_LIGHTNING ? silu_f(q[x]) : q[x]) * a.q_scale;
        }
        *reinterpret_cast<float4*>(v3) = make_float4(q[0], q[1], q[2], q[3]);
        *reinterpret_cast<float4*>(v3 + D) = make_float4(k[0], k[1], k[2], k[3]);
        if (OS_OWN_DECAY<MODE>) *reinterpret_cast<float4*>(v3 + 2 * D) = make_float4(w[0], w[1], w[2], w[3]);
      }
#pragma unroll
      for (int e = 0; e < VPT; ++e) {
        const int tt = (ht + e * RUN_STAGE) / OS_COLS, at = buf * C * OS_COLS + ht + e * RUN_STAGE;
        if (tt < nt) vcol[at] = GATES ? pv[e] * gate[2 * tt + 1] : MODE == OUTER_SCAN_LIGHTNING ? silu_f(pv[e]) : pv[e];
        if (MODE == OUTER_SCAN_SSD) vraw[at] = pv[e];
      }
    };
    auto normalise = [&](int n) {                    // GATED: n q of the chunk's tokens, a row per thread
      const int nt = min(C, sq.q_len - n * C);
      const float* gate = &gates[block_of(n)][n * C % 32][0];
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int i = ht + r * RUN_STAGE;
        if (i >= D) continue;
        float* v3 = vec + (size_t)(n % RING) * C * NV * D + i;
        float nk[C], q[C];
#pragma unroll
        for (int tt = 0; tt < C; ++tt) nk[tt] = gate[2 * tt + 1] * v3[tt * NV * D + D], q[tt] = v3[tt * NV * D];   // (behind the last token: not used)
#pragma unroll
        for (int tt = 0; tt < C; ++tt)
          if (tt < nt) {
            n_row[r] = fmaf(gate[2 * tt], n_row[r], nk[tt]);
            v3[tt * NV * D + 2 * D] = n_row[r] * q[tt];
          }
      }
    };
    const int n_blocks = (sq.q_len + 31) / 32;
    const bool first_warp = ht < 32;
    if (n_chunks > 0) fetch(0);
    if (GATES && first_warp) {
      fetch_gates(0);
      take_gates(0);
      fetch_gates(1);
    }
    for (int n = 0; n < n_chunks; ++n) {
      if (n >= RING) bar_sync_at<EMPTY>(n % RING, RUN_STAGE + RUN_WRITE);
      if (GATES) bar_sync_at<STAGED>(0, RUN_STAGE);  // the gates of this chunk's block are there
      stage(n);
      if (n + 1 < n_chunks) fetch(n + 1);
      if (MODE == OUTER_SCAN_GATED) {
        bar_sync_at<STAGED>(0, RUN_STAGE);           // every key of the chunk is there
        normalise(n);
      }
      bar_arrive_at<FULL>(n % RING, RUN_ROWS + RUN_STAGE);
      if (GATES && first_warp && n * C % 32 == 0 && n * C / 32 + 1 < n_blocks) {   // (the chunks of the block it replaces are out: EMPTY above)
        take_gates(n * C / 32 + 1);
        fetch_gates(n * C / 32 + 2);
      }
    }
  } else {
    // ===================== outputs: token t of a chunk by writer warp t & 1 =====================
    constexpr int TPW = C / 2;
    const int w = (ht - RUN_STAGE) >> 5;
    const float ssd_skip = MODE == OUTER_SCAN_SSD ? a.D[h] : 0.f;
    float* o_at = a.out + (size_t)(sq.q_start + w) * a.ldo + (size_t)h * a.vdim + c0 + lane;
    const bool o_in = c0 + lane < a.vdim;
    for (int n = 0; n < n_chunks; ++n) {
      const int buf = n % RING, nt = min(C, sq.q_len - n * C);
      bar_sync_at<DONE>(buf, RUN_ROWS + RUN_WRITE);
      float sum[TPW], d[TPW];
#pragma unroll
      for (int e = 0; e < TPW; ++e) {
        const int tt = w + 2 * e;
        const float* from = part + (size_t)(buf * C + tt) * OS_GROUPS * OS_COLS + lane;
        sum[e] = 0.f;
#pragma unroll
        for (int r = 0; r < OS_GROUPS; ++r) sum[e] += from[r * OS_COLS];
        d[e] = 0.f;
        if (MODE == OUTER_SCAN_GATED) {
#pragma unroll
          for (int i = 0; i < D; i += 32) d[e] += vec[((size_t)(buf * C + tt) * NV + 2) * D + i + lane];
        }
      }
      if (MODE == OUTER_SCAN_GATED) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int e = 0; e < TPW; ++e) d[e] += __shfl_xor_sync(0xffffffffu, d[e], o);
      }
#pragma unroll
      for (int e = 0; e < TPW; ++e) {
        const int tt = w + 2 * e;
        if (MODE == OUTER_SCAN_GATED) sum[e] = sum[e] / (fmaxf(fabsf(d[e]), floor_m[block_of(n)][n * C % 32 + tt]) + 1e-6f);
        if (MODE == OUTER_SCAN_SSD) sum[e] = fmaf(ssd_skip, vraw[(buf * C + tt) * OS_COLS + lane], sum[e]);
      }
      if (n + RING < n_chunks) bar_arrive_at<EMPTY>(buf, RUN_STAGE + RUN_WRITE);
#pragma unroll
      for (int e = 0; e < TPW; ++e)
        if (o_in && w + 2 * e < nt) o_at[(size_t)(2 * e) * a.ldo] = sum[e];
      o_at += (size_t)C * a.ldo;
    }
  }
  if (MODE == OUTER_SCAN_GATED) {                    // as above: the head's last piece overwrites what all of them started from
    __syncthreads();
    if (tid == 0) {
      int32_t* done = a.done + (size_t)slot * a.heads + h;
      last_block = nz == 1 || atomicAdd(done, 1) == nz - 1;
      if (last_block && nz > 1) *done = 0;
    }
    __syncthreads();
    if (last_block && ht >= 0 && ht < RUN_STAGE) {
#pragma unroll
      for (int r = 0; r < NR; ++r)
        if (ht + r * RUN_STAGE < D) a.n[((size_t)slot * a.heads + h) * D + ht + r * RUN_STAGE] = n_row[r];
      if (ht == 0) a.m[(size_t)slot * a.heads + h] = m_run;
    }
  }
  if (zb == 0 && h == 0 && a.x_last != nullptr) {
    const float* src = a.x + (size_t)(sq.q_start + sq.q_len - 1) * a.width;
    for (int i = tid; i < a.width; i += RUN_THREADS) a.x_last[(size_t)slot * a.width + i] = src[i];
  }
}

// Steps whose portions are single tokens: the same update and the same sums in the same order (bit for bit), laid out for the
// bytes of the state, which are all there is: 256 threads = 8 warps of rows x 32 lanes of CPT neighbouring columns, a whole
// [dim, 32 CPT] piece of a head requested at once, its lines already while the kernel before still runs.  Needs dim = 8 RPT and
// whole pieces.  32 tokens: gated, 8 heads of 128 x 256 (67 MB moved), 30.0 -> 16.4 us; decayed, 32 heads of 64 x 64, 15.0 -> 8.5.
template <int RPT, int MODE, int CPT>
__global__ void __launch_bounds__(OS_THREADS)
outer_step_kernel(OuterScan a, const AttnSeq* __restrict__ seqs, const int32_t* __restrict__ tok_slot) {
  constexpr int D = RPT * OS_GROUPS, COLS = 32 * CPT;
  __shared__ __align__(16) float vec[3][D];   // q | k | w (GATED: n q)
  __shared__ float part[OS_GROUPS][COLS];
  __shared__ float gates[3];                  // the decay, the factor of the outer product, GATED: e^(-m)
  griddep_launch();
  const AttnSeq sq = seqs[blockIdx.x];        // (written by the host before the step, as the slots are)
  const int h = blockIdx.y, tid = threadIdx.x, g = tid >> 5, lane = tid & 31;
  const int hq = a.qk_heads > 0 ? h / (a.heads / a.qk_heads) : h;
  const int c0 = blockIdx.z * COLS, slot = tok_slot[sq.q_start];
  const bool fresh = sq.kv_len == 1;
  constexpr bool OWN_DECAY = MODE == OUTER_SCAN_DECAY || MODE == OUTER_SCAN_HGRN || MODE == OUTER_SCAN_GLA;
  auto row_of = [&](int j) { return 4 * (g + (j >> 2) * OS_GROUPS) + (j & 3); };
  float* Sg = a.S + (((size_t)slot * a.heads + h) * D) * a.vdim + c0 + lane * CPT;
  if (!fresh && lane * CPT % 32 == 0) {
#pragma unroll
    for (int j = 0; j < RPT; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(Sg + (size_t)row_of(j) * a.vdim));
  }
  griddep_wait();
  float S[RPT][CPT];
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
#pragma unroll
    for (int e = 0; e < CPT; ++e) S[j][e] = 0.f;
    if (!fresh) {
      const float* from = Sg + (size_t)row_of(j) * a.vdim;
      if constexpr (CPT == 4) {
        ld_vec<4>(from, S[j]);
      } else {
        const float2 v = *reinterpret_cast<const float2*>(from);
        S[j][0] = v.x; S[j][1] = v.y;
      }
    }
  }
  const size_t row = (size_t)sq.q_start;
  float n_row = 0.f, m_run = 0.f;
  if (MODE == OUTER_SCAN_GATED && !fresh) {
    n_row = tid < D ? a.n[((size_t)slot * a.heads + h) * D + tid] : 0.f;
    m_run = a.m[(size_t)slot * a.heads + h];
  }
  if (tid < D) {
    const float q = a.q[row * a.ldq + (size_t)hq * D + tid];
    const float k = MODE == OUTER_SCAN_HGRN ? a.u[(size_t)h * D + tid] : a.k[row * a.ldk + (size_t)hq * D + tid];
    const float d = OWN_DECAY ? a.decay_raw[row * a.ldd + (size_t)h * D + tid] : 0.f, w = OWN_DECAY ? a.w0[(size_t)h * D + tid] : 0.f;
    if (MODE == OUTER_SCAN_HGRN) {
      vec[0][tid] = silu_f(q) * a.q_scale;
      vec[1][tid] = (1.f - k) * sigmoid_f(-(d + w));
      vec[2][tid] = k + (1.f - k) * sigmoid_f(d + w);
    } else if (MODE == OUTER_SCAN_LIGHTNING) {
      vec[0][tid] = silu_f(q) * a.q_scale;
      vec[1][tid] = silu_f(k);
    } else {
      vec[0][tid] = q * a.q_scale;
      vec[1][tid] = k;
      if (MODE == OUTER_SCAN_DECAY) vec[2][tid] = expf(-expf(d + w));
      if (MODE == OUTER_SCAN_GLA) vec[2][tid] = expf(logsigmoid_f(d + w) * a.inv_tau);
    }
  }
  float m_new = 0.f;
  if (MODE == OUTER_SCAN_GATED && tid == 0) {
    const float ig = a.gate_cap * tanhf((a.ig[row * a.ldg + h] + a.ig_b[h]) / a.gate_cap);
    const float fg = logsigmoid_f(a.gate_cap * tanhf((a.fg[row * a.ldg + h] + a.fg_b[h]) / a.gate_cap));
    m_new = fmaxf(fg + m_run, ig);
    gates[0] = expf(fg + m_run - m_new);
    gates[1] = expf(ig - m_new);
    gates[2] = expf(-m_new);
  }
  if (MODE == OUTER_SCAN_SSD && tid == 0) {
    const float dt = softplus_f(a.step_raw[row * a.lds + h] + a.step_b[h]);
    gates[0] = expf(-expf(a.A_log[h]) * dt);
    gates[1] = dt;
  }
  float vr[CPT];   // as it is (SSD's skip reads it), and times the gate
#pragma unroll
  for (int e = 0; e < CPT; ++e) {
    vr[e] = a.v[row * a.ldv + (size_t)h * a.vdim + c0 + lane * CPT + e];
    if (MODE == OUTER_SCAN_LIGHTNING) vr[e] = silu_f(vr[e]);
  }
  __syncthreads();
  if (MODE == OUTER_SCAN_GATED) {
    if (tid < D) {
      n_row = fmaf(gates[0], n_row, gates[1] * vec[1][tid]);
      vec[2][tid] = n_row * vec[0][tid];
    }
  }
  float wd = (MODE == OUTER_SCAN_LIGHTNING || MODE == OUTER_SCAN_RETENTION) ? a.decay[h] : 0.f, vc[CPT];
#pragma unroll
  for (int e = 0; e < CPT; ++e) vc[e] = vr[e];
  if (MODE == OUTER_SCAN_SSD || MODE == OUTER_SCAN_GATED) {
    wd = gates[0];
#pragma unroll
    for (int e = 0; e < CPT; ++e) vc[e] *= gates[1];
  }
  float o[CPT][4];
#pragma unroll
  for (int e = 0; e < CPT; ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[e][i] = 0.f;
#pragma unroll
  for (int j = 0; j < RPT; j += 4) {
    float q4[4], k4[4], w4[4] = {wd, wd, wd, wd}, u4[4] = {0.f, 0.f, 0.f, 0.f};
    const int i0 = row_of(j);
    ld_vec<4>(&vec[0][i0], q4);
    ld_vec<4>(&vec[1][i0], k4);
    if (OWN_DECAY) ld_vec<4>(&vec[2][i0], w4);
    if (MODE == OUTER_SCAN_DECAY) {
#pragma unroll
      for (int i = 0; i < 4; ++i) u4[i] = a.u[(size_t)h * D + i0 + i];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < CPT; ++e) {
        float& s = S[j + i][e];
        const float kv = __fmul_rn(k4[i], vc[e]);   // (rounded before it is added, as the packed product above is)
        if (MODE == OUTER_SCAN_DECAY) {
          o[e][i] = fmaf(q4[i], fmaf(u4[i], kv, s), o[e][i]);
          s = fmaf(w4[i], s, kv);
        } else {
          s = fmaf(w4[i], s, kv);
          o[e][i] = fmaf(q4[i], s, o[e][i]);
        }
      }
  }
#pragma unroll
  for (int e = 0; e < CPT; ++e) part[g][lane * CPT + e] = (o[e][0] + o[e][1]) + (o[e][2] + o[e][3]);
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    float* to = Sg + (size_t)row_of(j) * a.vdim;
    if constexpr (CPT == 4) *reinterpret_cast<float4*>(to) = make_float4(S[j][0], S[j][1], S[j][2], S[j][3]);
    else *reinterpret_cast<float2*>(to) = make_float2(S[j][0], S[j][1]);
  }
  __syncthreads();
  if (tid < COLS) {
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < OS_GROUPS; ++r) sum += part[r][tid];
    if (MODE == OUTER_SCAN_GATED) {
      float d = 0.f;
      for (int i = lane; i < D; i += 32) d += vec[2][i];
      d = warp_sum_f(d);
      sum = sum / (fmaxf(fabsf(d), gates[2]) + 1e-6f);
    }
    if (MODE == OUTER_SCAN_SSD) sum = fmaf(a.D[h], a.v[row * a.ldv + (size_t)h * a.vdim + c0 + tid], sum);
    a.out[row * a.ldo + (size_t)h * a.vdim + c0 + tid] = sum;
  }
  if (MODE == OUTER_SCAN_GATED) {   // as above: the head's last piece overwrites what all of them started from
    __shared__ int last_block;
    if (tid == 0) {
      int32_t* done = a.done + (size_t)slot * a.heads + h;
      last_block = gridDim.z == 1 || atomicAdd(done, 1) == (int)gridDim.z - 1;
      if (last_block && gridDim.z > 1) *done = 0;
    }
    __syncthreads();
    if (last_block) {
      if (tid < D) a.n[((size_t)slot * a.heads + h) * D + tid] = n_row;
      if (tid == 0) a.m[(size_t)slot * a.heads + h] = m_new;
    }
  }
  if (blockIdx.z == 0 && h == 0 && a.x_last != nullptr) {
    const float* src = a.x + row * a.width;
    for (int i = tid; i < a.width; i += OS_THREADS) a.x_last[(size_t)slot * a.width + i] = src[i];
  }
}

// ------------------------------------------------------------------------------------------------ convolution state
// grid (sequences, ceil(n / 128)): one thread per channel moves the tail of its convolution forward
__global__ void __launch_bounds__(128)
conv_state_save_kernel(const float* __restrict__ x, int ld, int n, int taps, const AttnSeq* __restrict__ seqs,
                       const int32_t* __restrict__ tok_slot, float* __restrict__ conv_state) {
  griddep_launch();
  griddep_wait();
  const AttnSeq sq = seqs[blockIdx.x];
  const int c = blockIdx.y * 128 + threadIdx.x;
  if (c >= n) return;
  const int K1 = taps - 1, first = sq.kv_len - sq.q_len, slot = tok_slot[sq.q_start];
  float* cs = conv_state + (size_t)slot * K1 * n + c;
  for (int e = 0; e < K1; ++e) {   // ascending: entry e + q_len is read before it could be rewritten
    const int pp = sq.kv_len - K1 + e;
    float v = 0.f;
    if (pp >= first) v = x[(size_t)(sq.q_start + pp - first) * ld + c];
    else if (pp >= 0) v = cs[(size_t)(e + sq.q_len) * n];
    cs[(size_t)e * n] = v;
  }
}

// ------------------------------------------------------------------------------------------------ gated delta rule
// grid (sequences, heads, ceil(vdim / 32)); 256 threads = 32 value columns x DS_LPC lanes.  A column of S is independent of
// the others (its write u_c needs only its own S[:, c] . k), so DS_LPC neighbouring lanes share one column, lane `sub` keeping
// rows 32 jj + 4 sub + (0..3) in registers; the two sums over the rows that a token needs -- (g S)[:, c] . k for the write and
// (g S)[:, c] . q for the read-out, which with the write becomes o_c = (g S)[:, c] . q + u_c (k . q) -- meet through one round of
// shuffles.  Normalised q / k, the decays and the per-token scalars are staged in shared memory DS_CHUNK tokens at a time (rows
// padded to a multiple of four with zeros, so a lane fetches its four rows of each vector with one 16-byte load); the token
// loop itself runs without a barrier.
constexpr int DS_LPC = 8, DS_COLS = 32, DS_THREADS = DS_LPC * DS_COLS, DS_CHUNK = 16;
template <int RPT>
__global__ void __launch_bounds__(DS_THREADS)
delta_scan_kernel(DeltaScan a, const AttnSeq* __restrict__ seqs, const int32_t* __restrict__ tok_slot) {
  extern __shared__ __align__(16) float ds_smem[];
  static_assert(RPT % 4 == 0, "a lane owns whole groups of four rows");
  const int D = a.dim, Dp = (D + 3) & ~3;
  float* vec = ds_smem;                                  // [DS_CHUNK][3][Dp]: q | k | decay
  float* vcol = vec + (size_t)DS_CHUNK * 3 * Dp;         // [DS_CHUNK][DS_COLS]
  __shared__ float beta_s[DS_CHUNK], kq_s[DS_CHUNK];
  griddep_launch();
  griddep_wait();
  const AttnSeq sq = seqs[blockIdx.x];
  const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sub = lane & (DS_LPC - 1);
  const int hq = h / (a.heads / a.qk_heads);
  const int cl = warp * (32 / DS_LPC) + lane / DS_LPC;   // column inside the CTA's 32
  const int c = blockIdx.z * DS_COLS + cl;
  const bool col_ok = c < a.vdim;
  const int slot = tok_slot[sq.q_start];
  const bool fresh = sq.kv_len - sq.q_len == 0;
  float S[RPT];
  float* Sg = a.S + (((size_t)slot * a.heads + h) * D) * a.vdim + (col_ok ? c : 0);
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int i = (j >> 2) * 32 + sub * 4 + (j & 3);
    S[j] = (!fresh && col_ok && i < D) ? Sg[(size_t)i * a.vdim] : 0.f;
  }
  const float rate = -expf(a.A_log[h]), q_mult = 1.f / sqrtf((float)D);
  // A chunk's raw values travel global memory -> registers -> shared memory: all loads of a chunk are issued back to back
  // (one round trip to memory, not one per element), and the loads of chunk n + 1 are issued before the token loop of chunk n.
  // thread (tt = tid / 16, l = tid % 16) stages entries l, l + 16, ... of token tt's vectors, and two of the chunk's values
  constexpr int EPT = RPT / 2;   // 8 RPT rows at most, 16 threads per token
  constexpr int TPT = DS_THREADS / DS_CHUNK;
  static_assert(TPT == 16 && DS_CHUNK * DS_COLS == 2 * DS_THREADS, "staging map");
  const int st_tt = tid / TPT, st_l = tid % TPT;
  float pq[EPT], pk[EPT], pd[EPT], pv[2], pb = 0.f;
  auto fetch = [&](int t0) {
    const int nt = min(DS_CHUNK, sq.q_len - t0);
    const bool tok = st_tt < nt;
    const size_t row = (size_t)(sq.q_start + t0 + (tok ? st_tt : 0));
    const float* qr = a.q + row * a.ldq + (size_t)hq * D;
    const float* kr_ = a.k + row * a.ldk + (size_t)hq * D;
    const float* dr = a.decay_raw + row * a.ldd + (size_t)h * D;
    const float* db = a.decay_b + (size_t)h * D;
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const int i = st_l + e * TPT;
      const bool in = tok && i < D;
      pq[e] = in ? qr[i] : 0.f;
      pk[e] = in ? kr_[i] : 0.f;
      pd[e] = in ? dr[i] + db[i] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {   // value columns: token tt, columns 2 l + e
      const int col = blockIdx.z * DS_COLS + 2 * st_l + e;
      pv[e] = (tok && col < a.vdim) ? a.v[row * a.ldv + (size_t)h * a.vdim + col] : 0.f;
    }
    pb = tid < nt ? a.beta_raw[(size_t)(sq.q_start + t0 + tid) * a.ldb + h] : 0.f;
  };
  fetch(0);
  for (int t0 = 0; t0 < sq.q_len; t0 += DS_CHUNK) {
    const int nt = min(DS_CHUNK, sq.q_len - t0);
    __syncthreads();   // the previous chunk's vectors are consumed
    if (st_tt < nt) {
      float* v3 = vec + (size_t)st_tt * 3 * Dp;
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const int i = st_l + e * TPT;
        if (i < Dp) {
          v3[i] = pq[e];
          v3[Dp + i] = pk[e];
          v3[2 * Dp + i] = i < D ? expf(rate * softplus_f(pd[e])) : 0.f;
        }
      }
    }
    vcol[st_tt * DS_COLS + 2 * st_l] = pv[0];
    vcol[st_tt * DS_COLS + 2 * st_l + 1] = pv[1];
    if (tid < nt) beta_s[tid] = sigmoid_f(pb);
    __syncthreads();
    if (t0 + DS_CHUNK < sq.q_len) fetch(t0 + DS_CHUNK);   // lands while this chunk's tokens are worked through
    for (int tt = warp; tt < nt; tt += DS_THREADS / 32) {   // unit vectors, and k . q of the unit vectors
      float* v3 = vec + (size_t)tt * 3 * Dp;
      float sq2 = 0.f, sk2 = 0.f, skq = 0.f;
      for (int i = lane; i < D; i += 32) {
        const float qv = v3[i], kv = v3[Dp + i];
        sq2 = fmaf(qv, qv, sq2); sk2 = fmaf(kv, kv, sk2); skq = fmaf(qv, kv, skq);
      }
      sq2 = warp_sum_f(sq2); sk2 = warp_sum_f(sk2); skq = warp_sum_f(skq);
      const float rq = q_mult / sqrtf(sq2 + 1e-6f), rk = 1.f / sqrtf(sk2 + 1e-6f);
      for (int i = lane; i < D; i += 32) { v3[i] *= rq; v3[Dp + i] *= rk; }
      if (lane == 0) kq_s[tt] = skq * rq * rk;
    }
    __syncthreads();
    const float* v3 = vec;
    for (int tt = 0; tt < nt; ++tt, v3 += 3 * Dp) {
      float kr[RPT];
      float sk = 0.f, sqv = 0.f;
#pragma unroll
      for (int jj = 0; jj < RPT / 4; ++jj) {
        const int i0 = jj * 32 + sub * 4;
        if (i0 < Dp) {
          const float4 q4 = *reinterpret_cast<const float4*>(v3 + i0);
          const float4 k4 = *reinterpret_cast<const float4*>(v3 + Dp + i0);
          const float4 g4 = *reinterpret_cast<const float4*>(v3 + 2 * Dp + i0);
          const float qa[4] = {q4.x, q4.y, q4.z, q4.w}, ka[4] = {k4.x, k4.y, k4.z, k4.w}, ga[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int j = jj * 4 + e;
            S[j] *= ga[e];
            sk = fmaf(S[j], ka[e], sk);
            sqv = fmaf(S[j], qa[e], sqv);
            kr[j] = ka[e];
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) kr[jj * 4 + e] = 0.f;
        }
      }
#pragma unroll
      for (int o = DS_LPC / 2; o > 0; o >>= 1) {
        sk += __shfl_xor_sync(0xffffffffu, sk, o);
        sqv += __shfl_xor_sync(0xffffffffu, sqv, o);
      }
      const float u = beta_s[tt] * (vcol[tt * DS_COLS + cl] - sk);
#pragma unroll
      for (int j = 0; j < RPT; ++j) S[j] = fmaf(kr[j], u, S[j]);
      if (sub == 0 && col_ok) a.out[(size_t)(sq.q_start + t0 + tt) * a.ldo + (size_t)h * a.vdim + c] = fmaf(u, kq_s[tt], sqv);
    }
  }
  if (col_ok) {
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int i = (j >> 2) * 32 + sub * 4 + (j & 3);
      if (i < D) Sg[(size_t)i * a.vdim] = S[j];
    }
  }
}

// ------------------------------------------------------------------------------------------------ head norm + gate
// grid (T, ceil(heads / 4)), 128 threads: one warp per (token, head)
__global__ void __launch_bounds__(128)
head_norm_gate_kernel(const float* __restrict__ o, int ldo, int heads, int vdim, const float* __restrict__ w,
                      const float* __restrict__ gate, int ldg, int act, float eps, void* __restrict__ out, int out_dtype,
                      int out_ld, int gate_first, float mult) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= heads) return;
  const float* orow = o + (size_t)t * ldo + (size_t)h * vdim;
  float ss = 0.f;
  if (gate_first) {   // the gated values are what is normed
    const float* grow = gate + (size_t)t * ldg + (size_t)h * vdim;
    for (int i = lane; i < vdim; i += 32) {
      const float v = orow[i] * (act == 1 ? silu_f(grow[i]) : sigmoid_f(grow[i]));
      ss = fmaf(v, v, ss);
    }
    const float rs = 1.f / sqrtf(warp_sum_f(ss) / (float)vdim + eps);
    for (int i = lane; i < vdim; i += 32) {
      const float v = orow[i] * (act == 1 ? silu_f(grow[i]) : sigmoid_f(grow[i]));
      st_op(out, out_dtype, (size_t)t * out_ld + (size_t)h * vdim + i, v * rs * (w != nullptr ? w[(size_t)h * vdim + i] : 1.f) * mult);
    }
    return;
  }
  for (int i = lane; i < vdim; i += 32) ss = fmaf(orow[i], orow[i], ss);
  const float rs = 1.f / sqrtf(warp_sum_f(ss) / (float)vdim + eps);
  for (int i = lane; i < vdim; i += 32) {
    float gv = 1.f;
    if (act != 2) {
      const float gl = gate[(size_t)t * ldg + (size_t)h * vdim + i];
      gv = act == 1 ? silu_f(gl) : sigmoid_f(gl);
    }
    st_op(out, out_dtype, (size_t)t * out_ld + (size_t)h * vdim + i, orow[i] * rs * (w != nullptr ? w[(size_t)h * vdim + i] : 1.f) * (gv * mult));
  }
}

// the same for heads of a multiple of four values (<= 512) whose rows start on 16-byte boundaries: four values per lane and step, kept
// in registers between the two passes
constexpr int HNG_V = 4;
__global__ void __launch_bounds__(128)
head_norm_gate_vec_kernel(const float* __restrict__ o, int ldo, int heads, int vdim, const float* __restrict__ w,
                          const float* __restrict__ gate, int ldg, int act, float eps, void* __restrict__ out, int out_dtype,
                          int out_ld, float mult) {
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= heads) return;
  const float* orow = o + (size_t)t * ldo + (size_t)h * vdim;
  const float* grow = act != 2 ? gate + (size_t)t * ldg + (size_t)h * vdim : nullptr;
  float4 v[HNG_V], g[HNG_V];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < HNG_V; ++j) {
    const int i = (j * 32 + lane) * 4;
    v[j] = i < vdim ? *reinterpret_cast<const float4*>(orow + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (grow != nullptr && i < vdim) g[j] = *reinterpret_cast<const float4*>(grow + i);
    ss = fmaf(v[j].x, v[j].x, fmaf(v[j].y, v[j].y, fmaf(v[j].z, v[j].z, fmaf(v[j].w, v[j].w, ss))));
  }
  const float rs = mult / sqrtf(warp_sum_f(ss) / (float)vdim + eps);
#pragma unroll
  for (int j = 0; j < HNG_V; ++j) {
    const int i = (j * 32 + lane) * 4;
    if (i >= vdim) break;
    float r[4] = {v[j].x * rs, v[j].y * rs, v[j].z * rs, v[j].w * rs};
    if (w != nullptr) {
      const float4 x = *reinterpret_cast<const float4*>(w + (size_t)h * vdim + i);
      r[0] *= x.x; r[1] *= x.y; r[2] *= x.z; r[3] *= x.w;
    }
    if (grow != nullptr) {
      const float z[4] = {g[j].x, g[j].y, g[j].z, g[j].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) r[e] *= act == 1 ? silu_f(z[e]) : sigmoid_f(z[e]);
    }
    const size_t at = (size_t)t * out_ld + (size_t)h * vdim + i;
    if (out_dtype == DT_BF16) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(r[0], r[1]), hi = __floats2bfloat162_rn(r[2], r[3]);
      uint2 pk;
      pk.x = *reinterpret_cast<const uint32_t*>(&lo);
      pk.y = *reinterpret_cast<const uint32_t*>(&hi);
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(out) + at) = pk;
    } else {
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + at) = make_float4(r[0], r[1], r[2], r[3]);
    }
  }
}

// wide groups (a whole row normed as one or a few groups): grid (T, heads), 256 threads, one CTA per (token, group)
__global__ void __launch_bounds__(256)
head_norm_gate_wide_kernel(const float* __restrict__ o, int ldo, int heads, int vdim, const float* __restrict__ w,
                           const float* __restrict__ gate, int ldg, int act, float eps, void* __restrict__ out, int out_dtype,
                           int out_ld, int gate_first, float mult) {
  __shared__ float red[8];
  griddep_launch();
  griddep_wait();
  const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const float* orow = o + (size_t)t * ldo + (size_t)h * vdim;
  const float* grow = gate + (size_t)t * ldg + (size_t)h * vdim;
  float ss = 0.f;
  for (int i = tid; i < vdim; i += 256) {
    float v = orow[i];
    if (gate_first && act != 2) v *= act == 1 ? silu_f(grow[i]) : sigmoid_f(grow[i]);
    ss = fmaf(v, v, ss);
  }
  ss = warp_sum_f(ss);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int r = 0; r < 8; ++r) tot += red[r];   // the same order in every thread
  const float rs = 1.f / sqrtf(tot / (float)vdim + eps);
  for (int i = tid; i < vdim; i += 256) {
    const float gv = act == 2 ? 1.f : act == 1 ? silu_f(grow[i]) : sigmoid_f(grow[i]);
    st_op(out, out_dtype, (size_t)t * out_ld + (size_t)h * vdim + i, orow[i] * gv * rs * (w != nullptr ? w[(size_t)h * vdim + i] : 1.f) * mult);
  }
}

__global__ void convert_f32_kernel(const float* __restrict__ x, void* __restrict__ out, int out_dtype, size_t n) {
  griddep_launch();
  griddep_wait();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    st_op(out, out_dtype, i, x[i]);
}

}  // namespace

cudaError_t token_shift_mix_launch(const float* x, int width, const float* mu, int n_mix, const int32_t* positions,
                                   const int32_t* tok_slot, const float* prev_state, void* out, int out_dtype,
                                   long long out_bs, int T, cudaStream_t stream) {
  if (T <= 0) return cudaSuccess;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (width % 4 == 0 && out_bs % 4 == 0 && al16(x) && al16(mu) && al16(prev_state) && al16(out))
    return launch_k(token_shift_mix_kernel<4>, dim3(T, (width / 4 + 127) / 128), dim3(128), 0, stream, x, width, mu, n_mix, positions,
                    tok_slot, prev_state, out, out_dtype, out_bs);
  return launch_k(token_shift_mix_kernel<1>, dim3(T, (width + 127) / 128), dim3(128), 0, stream, x, width, mu, n_mix, positions, tok_slot,
                  prev_state, out, out_dtype, out_bs);
}

cudaError_t short_conv_silu_launch(const float* xz, int ld, int inner, const float* w, const float* b, int taps,
                                   const int32_t* positions, const int32_t* tok_slot, const float* conv_state,
                                   float* out_f32, void* out_op, int out_dtype, int T, cudaStream_t stream) {
  if (T <= 0) return cudaSuccess;
  if (taps < 1) return cudaErrorInvalidValue;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (ld % 4 == 0 && inner % 4 == 0 && al16(xz) && al16(conv_state) && al16(out_f32) && al16(w) && al16(out_op)) {
    if (taps == 4 && T >= 256)   // (blocks enough with eight tokens each)
      return launch_k(short_conv_run_kernel, dim3((T + CONV_RUN - 1) / CONV_RUN, (inner / 4 + 127) / 128), dim3(128), 0, stream, xz, ld, inner, w, b,
                      positions, tok_slot, conv_state, out_f32, out_op, out_dtype, T);
    return launch_k(short_conv_silu_kernel<4>, dim3(T, (inner / 4 + 127) / 128), dim3(128), 0, stream, xz, ld, inner, w, b, taps,
                    positions, tok_slot, conv_state, out_f32, out_op, out_dtype);
  }
  return launch_k(short_conv_silu_kernel<1>, dim3(T, (inner + 127) / 128), dim3(128), 0, stream, xz, ld, inner, w, b, taps,
                  positions, tok_slot, conv_state, out_f32, out_op, out_dtype);
}

// Tokens of a chunk: sixteen for long portions, whose tokens' latency is what is bound; fewer where portions end inside their first chunks, or
// where the blocks fill the chip several times over and eight tokens' registers let more of them in.  4096 channels of 16 states,
// microseconds, chunks of 16 / 8 / 4: one portion of 1024 tokens 119 / 152 / -, 20 of 100 138 / 127 / 128, 32 of 16 44 / 36 / 36, 64 of 5 85 / 41 /
// 37, 128 of 2 115 / 68 / 47, one of 200 beside 31 of 5 55 / 43 / 48; 256 channels, one of 128 beside 31 of 1 18 / 21 / 25.  (Before there were
// chunks of 16 and branches out of the token loop: 282, 150, 43, 40, 61, 90; 36.)  Of fewer states chunks of eight are behind those of four.
static int scan_chunk(const SelScan& a, int n_seqs, long long blocks) {
  if (a.longest <= 0 || a.longest >= 256) return 16;
  if (blocks <= 16 * 148) return a.longest >= 48 ? 16 : a.longest >= 7 ? 8 : 4;
  return a.tokens >= 8 * n_seqs ? 8 : 4;
}
cudaError_t selective_scan_launch(const SelScan& a, const AttnSeq* seqs, int n_seqs, const int32_t* tok_slot,
                                  cudaStream_t stream) {
  if (n_seqs <= 0) return cudaSuccess;
  if (a.state < 1 || a.state > SELSCAN_MAX_STATE || a.taps < 1) return cudaErrorInvalidValue;
  const size_t bc = (size_t)SCAN_CHUNK * 2 * a.state * sizeof(float);
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (a.single && a.state == SCAN_REG_STATE && al16(a.S) && al16(a.A_log))
    return launch_k(selective_step_kernel, dim3(n_seqs, (a.inner + 63) / 64), dim3(256), 0, stream, a, seqs, tok_slot);
  if (a.state <= SCAN_REG_STATE) {
    constexpr int per_cta = SCAN_THREADS / SCAN_LPC;
    const long long blocks = (long long)n_seqs * ((a.inner + per_cta - 1) / per_cta);
    if (blocks >= (1ll << 31)) return cudaErrorInvalidValue;
    const bool all = a.state == SCAN_REG_STATE;
    const int chunk = scan_chunk(a, n_seqs, blocks);
    const auto kernel = chunk == 16 ? (all ? selective_scan_reg_kernel<true, 16> : selective_scan_reg_kernel<false, 16>)
                      : chunk == 8 && all ? selective_scan_reg_kernel<true, 8>
                      : all ? selective_scan_reg_kernel<true, 4> : selective_scan_reg_kernel<false, 4>;
    return launch_k(kernel, dim3((unsigned)blocks), dim3(SCAN_THREADS), 0, stream, a, seqs, n_seqs, tok_slot);
  }
  const dim3 grid(n_seqs, (a.inner + SCAN_THREADS - 1) / SCAN_THREADS);
  const size_t smem = bc + (size_t)2 * a.state * SCAN_THREADS * sizeof(float);
  static size_t smem_set = 0;
  if (smem > 48 * 1024 && smem > smem_set) {
    const cudaError_t e = cudaFuncSetAttribute(selective_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    smem_set = smem;
  }
  return launch_k(selective_scan_kernel, grid, dim3(SCAN_THREADS), smem, stream, a, seqs, tok_slot);
}

// Steps that run in outer_run_kernel.  It works a long portion through in half the time, but takes twice the time to begin and end one: of
// few portions it is ahead from 16 or 17 tokens on (44 with keys of more than 128 rows and where the gate writes the key).  Where the pieces
// fill the chip several times over it is from 28 on, and what many short portions lose outweighs the chain of one long one unless that is
// twice as long as there are portions, or the portions are long on average.  Gated memory of 8 heads of 128 x 256, microseconds, outer_scan_kernel / here: 128
// portions of 2 tokens 87 / 167, 32 of 16 43 / 51, of 32 75 / 74, of 64 143 / 124; one of 128 beside 31 of 1 60 / 48, of 64 beside 60 of 4
// 62 / 82, of 100 beside 100 of 1 90 / 158.  One portion of 17 tokens 8.8 / 8.6, of 24 9.9 / 8.8, three of 3 5.7 / 7.6; 32 decayed heads of 64 x 64,
// one portion of 17 5.4 / 4.7; keys that the gate writes, 8 heads of 128 x 128, one portion of 28 10.4 / 12.1.
template <int RPT, int MODE>
static bool outer_runs(const OuterScan& a, int n_seqs, long long pieces) {
  constexpr bool slow = RPT > 16 || MODE == OUTER_SCAN_HGRN;
  constexpr int chip = 3 * 148 * (RPT <= 16 ? 2 : 1);
  if (a.longest <= 0) return true;
  if (pieces <= chip) return a.longest >= (slow ? 44 : 16);
  return a.longest >= (slow ? 44 : 28) && (a.longest >= 2 * n_seqs || a.tokens >= (RPT > 16 ? 80 : 40) * n_seqs);
}
template <int RPT, int MODE>
static cudaError_t outer_run(const OuterScan& a, const AttnSeq* seqs, int n_seqs, int pieces, const int32_t* tok_slot, cudaStream_t stream) {
  auto al16 = [](const float* p, int ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 4 == 0; };   // (nullptr where the mode has none)
  const bool vec16 = al16(a.q, a.ldq) && (MODE == OUTER_SCAN_HGRN || al16(a.k, a.ldk)) && (!OS_OWN_DECAY<MODE> || al16(a.decay_raw, a.ldd));
  auto launch = [&](auto kernel, cudaError_t attr) {
    if (attr != cudaSuccess) return attr;
    return launch_k(kernel, dim3(pieces), dim3(RUN_THREADS), RUN_SMEM<RPT, MODE>, stream, a, seqs, n_seqs, tok_slot);
  };
  auto room = [](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RUN_SMEM<RPT, MODE>); };
  if (vec16) {
    static const cudaError_t attr = room(outer_run_kernel<RPT, MODE, true>);
    return launch(outer_run_kernel<RPT, MODE, true>, attr);
  }
  static const cudaError_t attr = room(outer_run_kernel<RPT, MODE, false>);
  return launch(outer_run_kernel<RPT, MODE, false>, attr);
}
template <int RPT, int MODE>
static cudaError_t outer_scan_rows(const OuterScan& a, const AttnSeq* seqs, int n_seqs, const int32_t* tok_slot, cudaStream_t stream) {
  if constexpr (RPT <= 16) {   // (more rows, and columns that are no whole pieces, have no step kernel: 32 x 4 state values would spill)
    if (a.single && a.dim == RPT * OS_GROUPS && (reinterpret_cast<uintptr_t>(a.S) & 15) == 0) {
      if (a.vdim % 128 == 0) return launch_k(outer_step_kernel<RPT, MODE, 4>, dim3(n_seqs, a.heads, a.vdim / 128), dim3(OS_THREADS), 0, stream, a, seqs, tok_slot);
      if (a.vdim % 64 == 0) return launch_k(outer_step_kernel<RPT, MODE, 2>, dim3(n_seqs, a.heads, a.vdim / 64), dim3(OS_THREADS), 0, stream, a, seqs, tok_slot);
    }
  }
  const long long pieces = (long long)n_seqs * a.heads * ((a.vdim + OS_COLS - 1) / OS_COLS);
  if (a.dim == RPT * OS_GROUPS && pieces < (1ll << 31) && outer_runs<RPT, MODE>(a, n_seqs, pieces))
    return outer_run<RPT, MODE>(a, seqs, n_seqs, (int)pieces, tok_slot, stream);
  const dim3 grid(n_seqs, a.heads, (a.vdim + OS_COLS - 1) / OS_COLS);
  const size_t smem = ((size_t)OS_CHUNK * 3 * ((a.dim + 3) & ~3) + OS_CHUNK * OS_COLS) * sizeof(float);   // <= 50 KB (+ 17 KB static)
  const auto kernel = a.dim == RPT * OS_GROUPS ? outer_scan_kernel<RPT, MODE, true> : outer_scan_kernel<RPT, MODE, false>;
  if (RPT > 16) {   // keys of more than 128 entries: the staged chunk passes the default 48 KB of shared memory
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    if (e != cudaSuccess) return e;
  }
  return launch_k(kernel, grid, dim3(OS_THREADS), smem, stream, a, seqs, tok_slot);
}
template <int MODE>
static cudaError_t outer_scan_mode(const OuterScan& a, const AttnSeq* seqs, int n_seqs, const int32_t* tok_slot,
                                   cudaStream_t stream) {
  if (a.dim <= 8 * OS_GROUPS) return outer_scan_rows<8, MODE>(a, seqs, n_seqs, tok_slot, stream);
  if (a.dim <= 16 * OS_GROUPS) return outer_scan_rows<16, MODE>(a, seqs, n_seqs, tok_slot, stream);
  return outer_scan_rows<32, MODE>(a, seqs, n_seqs, tok_slot, stream);
}
cudaError_t outer_scan_launch(const OuterScan& a, const AttnSeq* seqs, int n_seqs, const int32_t* tok_slot,
                              cudaStream_t stream) {
  if (n_seqs <= 0) return cudaSuccess;
  if (a.dim < 1 || a.dim > OUTER_SCAN_MAX_DIM || a.heads < 1 || a.heads > 65535 || a.vdim < 1) return cudaErrorInvalidValue;
  if (a.qk_heads > 0 && a.heads % a.qk_heads != 0) return cudaErrorInvalidValue;
  if (a.mode == OUTER_SCAN_SSD) {
    if (a.step_raw == nullptr || a.step_b == nullptr || a.A_log == nullptr || a.D == nullptr) return cudaErrorInvalidValue;
    return outer_scan_mode<OUTER_SCAN_SSD>(a, seqs, n_seqs, tok_slot, stream);
  }
  if (a.mode == OUTER_SCAN_LIGHTNING) {
    if (a.decay == nullptr) return cudaErrorInvalidValue;
    return outer_scan_mode<OUTER_SCAN_LIGHTNING>(a, seqs, n_seqs, tok_slot, stream);
  }
  if (a.mode == OUTER_SCAN_RETENTION) {
    if (a.decay == nullptr) return cudaErrorInvalidValue;
    return outer_scan_mode<OUTER_SCAN_RETENTION>(a, seqs, n_seqs, tok_slot, stream);
  }
  if (a.mode == OUTER_SCAN_GLA) {
    if (a.decay_raw == nullptr || a.w0 == nullptr || !(a.inv_tau > 0.f)) return cudaErrorInvalidValue;
    return outer_scan_mode<OUTER_SCAN_GLA>(a, seqs, n_seqs, tok_slot, stream);
  }
  if (a.mode == OUTER_SCAN_HGRN) {
    if (a.decay_raw == nullptr || a.w0 == nullptr || a.u == nullptr) return cudaErrorInvalidValue;
    return outer_scan_mode<OUTER_SCAN_HGRN>(a, seqs, n_seqs, tok_slot, stream);
  }
  if (a.mode == OUTER_SCAN_GATED && a.done == nullptr) return cudaErrorInvalidValue;
  return a.mode == OUTER_SCAN_GATED ? outer_scan_mode<OUTER_SCAN_GATED>(a, seqs, n_seqs, tok_slot, stream)
                                    : outer_scan_mode<OUTER_SCAN_DECAY>(a, seqs, n_seqs, tok_slot, stream);
}

cudaError_t head_norm_gate_launch(const float* o, int ldo, int heads, int vdim, const float* w, const float* gate,
                                  int ldg, int act, float eps, void* out, int out_dtype, int T, cudaStream_t stream,
                                  int gate_first, float mult, int out_ld) {
  if (T <= 0) return cudaSuccess;
  if (act == 2) gate_first = 0;
  else if (gate == nullptr) return cudaErrorInvalidValue;
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (out_ld <= 0) out_ld = heads * vdim;
  if (gate_first == 0 && vdim % 4 == 0 && vdim <= 128 * HNG_V && ldo % 4 == 0 && out_ld % 4 == 0 && al16(o) && al16(w) && al16(out) &&
      (act == 2 || (ldg % 4 == 0 && al16(gate))))
    return launch_k(head_norm_gate_vec_kernel, dim3(T, (heads + 3) / 4), dim3(128), 0, stream, o, ldo, heads, vdim, w, gate, ldg, act, eps,
                    out, out_dtype, out_ld, mult);
  if (vdim >= 1024 && heads <= 65535)
    return launch_k(head_norm_gate_wide_kernel, dim3(T, heads), dim3(256), 0, stream, o, ldo, heads, vdim, w, gate, ldg, act, eps, out,
                    out_dtype, out_ld, gate_first, mult);
  return launch_k(head_norm_gate_kernel, dim3(T, (heads + 3) / 4), dim3(128), 0, stream, o, ldo, heads, vdim, w, gate, ldg, act,
                  eps, out, out_dtype, out_ld, gate_first, mult);
}

cudaError_t conv_state_save_launch(const float* x, int ld, int n, int taps, const AttnSeq* seqs, int n_seqs,
                                   const int32_t* tok_slot, float* conv_state, cudaStream_t stream) {
  if (n_seqs <= 0 || taps <= 1) return cudaSuccess;
  return launch_k(conv_state_save_kernel, dim3(n_seqs, (n + 127) / 128), dim3(128), 0, stream, x, ld, n, taps, seqs, tok_slot,
                  conv_state);
}

template <int RPT>
static cudaError_t delta_scan_rpt(const DeltaScan& a, const AttnSeq* seqs, int n_seqs, const int32_t* tok_slot, cudaStream_t stream) {
  const dim3 grid(n_seqs, a.heads, (a.vdim + DS_COLS - 1) / DS_COLS);
  const size_t smem = ((size_t)DS_CHUNK * 3 * ((a.dim + 3) & ~3) + DS_CHUNK * DS_COLS) * sizeof(float);
  if (smem > 48 * 1024) {
    static bool attr_set = false;
    if (!attr_set) {
      const cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel<RPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
      if (e != cudaSuccess) return e;
      attr_set = true;
    }
  }
  return launch_k(delta_scan_kernel<RPT>, grid, dim3(DS_THREADS), smem, stream, a, seqs, tok_slot);
}
cudaError_t delta_scan_launch(const DeltaScan& a, const AttnSeq* seqs, int n_seqs, const int32_t* tok_slot,
                              cudaStream_t stream) {
  if (n_seqs <= 0) return cudaSuccess;
  if (a.dim < 1 || a.dim > DELTA_SCAN_MAX_DIM || a.heads < 1 || a.heads > 65535 || a.vdim < 1 || a.qk_heads < 1 ||
      a.heads % a.qk_heads != 0)
    return cudaErrorInvalidValue;
  if (a.dim <= 32) return delta_scan_rpt<4>(a, seqs, n_seqs, tok_slot, stream);
  if (a.dim <= 8 * DS_LPC) return delta_scan_rpt<8>(a, seqs, n_seqs, tok_slot, stream);
  if (a.dim <= 16 * DS_LPC) return delta_scan_rpt<16>(a, seqs, n_seqs, tok_slot, stream);
  return delta_scan_rpt<32>(a, seqs, n_seqs, tok_slot, stream);
}

cudaError_t convert_f32_launch(const float* x, void* out, int out_dtype, size_t n, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 8);
  return launch_k(convert_f32_kernel, dim3(blocks), dim3(256), 0, stream, x, out, out_dtype, n);
}

}  // namespace tgis
