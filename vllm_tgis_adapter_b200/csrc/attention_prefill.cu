// Causal attention of prompts and prompt portions over the paged cache, on tcgen05 (reference call site: grpc_server.py:222 ->
// vllm v1/attention/backends/flashinfer.py:1665).  GQA, head_dim 128, bf16 in, fp32 softmax.
//
// A unit of work is 2 x TM query tokens of one sequence and one kv head; the G query heads that share the kv head lie beside
// each other in the rows (row = token * G + head), so TM = 128 / G tokens (rounded down to a multiple of 8) fill one M = 128
// accumulator and both accumulators of the CTA read every K and V tile that was staged once.  One CTA per SM walks the
// units; the host lists them longest first and the CTAs take them in snake order.
//
// Cache tiles are 128 tokens.  The layouts of the cache are those of the tensor cores' operands, so nothing is rearranged:
//   K  [16 chunks of 8 dims][32 tok][8] is the unswizzled K-major form (8 tokens x 16 bytes are one core matrix); sixteen bulk
//      copies of 512 bytes put a block between its neighbours, [16 chunks][128 tok][8];
//   V  [32 tok][16 chunks ^ (tok & 7)][8], read as two halves of 64 dims, is the 128-byte swizzled MN-major form: one 3-D box.
// S = Q K^T goes to TMEM; a thread per row takes its 128 scores, leaves the probabilities in their place as bf16 high parts (64
// columns) and low parts (64 columns: 16 mantissa bits in all, so that the result tracks an fp32 softmax), and the tensor cores
// read them from there: O += P_hi V + P_lo V.  The two accumulators alternate, so one's softmax runs under the other's products.
// The running maximum a row's sums refer to moves only when a score exceeds it by 2^8 (the sums are in fp32, so nothing is
// lost below it); a warp scales its part of O only then (the conditional rescaling published with FlashAttention-4).  A row's bits
// depend on its own keys alone: tiles are counted from the sequence's first token, and what another row or request does changes
// neither order nor reference of its sums.  The one thing that reaches a row from a key it does not see is a value that is not
// finite: the tensor cores add 0 * V.  A row that comes out with such numbers although no key that it sees has them is summed again
// over its own keys alone (sum_again), without the matrix instructions: its bits are then those of another order, and its numbers right.
//
// What bounds it: the tensor pipe, 3 x 128 x 128 x 128 multiply-adds a tile (S once, P V twice) -- 56 % active on an SM that has work
// (1859 tokens behind 6144), the rest goes to the way S -> softmax -> P V of one accumulator where it is longer than the other's
// products -- and whole units: 2048 tokens are 256 of them, so some SMs work twice and some once.  Microseconds a launch on one B200, 32 query
// and 8 kv heads, against the mma.sync kernel that went before (16 tokens x one head a warp, 32-token blocks, its pipe 56 %
// active): 1859 tokens behind 6144: 1289 -> 345 (620 TFLOP/s, counting P V once); 2048 alone 243 -> 61; 2048 in 6 prompts 71 -> 30;
// 32 prompts of 64 tokens 21.7 -> 16.1; 96 of 9 to 56 33.3 -> 29.3.  No faster: two threads per row (345 -> 356, short prompts
// 29 -> 39), tiles of 64 tokens with scores two tiles ahead (404), P handed over in halves (344).
//
// One short prompt is a chain of latencies and of CTAs that wait for their SM: with two accumulators a CTA takes all of its registers and
// shared memory, so neither it nor the product behind it can be resident under the kernel before.  A step of at most 128 keys a sequence
// and one unit per SM (prefill_units_build) therefore has one accumulator per CTA and rings as long as its longest sequence; and of
// at most 32 keys 90 registers a thread, which is what fits beside a CTA of the product cut along k.  Microseconds of a whole prompt step,
// mma.sync kernel -> two accumulators -> this: 8 layers of the 8B model, 17 tokens 839 -> 867 -> 840, 32 tokens 867 -> 897 -> 874, 64 tokens
// 1019 -> 951 -> 917; 12 layers 768 wide, 17 tokens 364 -> 400 -> 378, 64 tokens 634 -> 686 -> 667 (the mma.sync kernel stays ahead there:
// its operands need no copy, barrier and commit each; but a row's bits would depend on its step if it took these).
//
// No wait is unbounded: after about two seconds a role gives up, raises the word that gemm_pair_failed() looks at and leaves;
// copies and MMAs in flight land first and TMEM is freed on every path.
#include <algorithm>

#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace tgis {
namespace {

// ACC accumulators: warps 0..3 softmax of accumulator 0, 4..7 of 1, then one for copies, one for MMAs, (ACC = 2) two idle
constexpr int PT_THREADS(int acc) { return acc == 2 ? 384 : 192; }
constexpr int PT_REGS_SOFTMAX = 208, PT_REGS_OTHER = 88; // 256 x 208 + 128 x 88 = 384 x 168, what the launch gives every thread
constexpr int PT_KV = 128;                               // tokens of a cache tile
constexpr int PT_BLOCKS = PT_KV / KV_BLOCK;
constexpr int PT_BLOCK_BYTES = KV_BLOCK * HEAD_DIM * 2;
constexpr int PT_TILE_BYTES = PT_KV * HEAD_DIM * 2;      // 32 KiB: a K tile, a V tile, one accumulator's Q
// Q, rings of ACC tiles of `blocks` cache blocks for K and V, barriers
constexpr size_t PT_SMEM(int acc, int blocks) { return (size_t)acc * (PT_TILE_BYTES + 2 * blocks * PT_BLOCK_BYTES) + 1024 + 256; }
constexpr float PT_SLACK = 8.f;                          // exp2 domain: how far a score may exceed its row's reference

struct PrefillArgs {
  const __nv_bfloat16 *qkv, *k_cache, *v_cache;
  const PrefillUnit* units;
  const int32_t* block_table;
  __nv_bfloat16* out;
  int n_units, bt_stride, qkv_ld, out_ld, n_kv, G, TM;
  int blocks;                                            // ACC = 1: of a tile (all keys of a unit)
  float sl2;                                             // |scale| * log2(e)
  uint32_t minus;                                        // scale < 0: bit "negate A" of the score products' descriptor
  int* err;
};

__device__ __forceinline__ void tma_load_3d(const CUtensorMap* m, uint64_t* bar, void* dst, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];\n" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// D (+)= A[tmem] B[smem]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)layout << 61;
}
__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t x, uint64_t y, uint64_t z) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x), "l"(y), "l"(z));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t x, uint64_t y) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t cvt2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <int N, bool UP>
__device__ __forceinline__ void set_regs() {
  if constexpr (UP) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
  else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
__device__ __forceinline__ bool bounded_wait(uint64_t* bar, uint32_t parity, int* err) {
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

struct Unit : PrefillUnit {
  int n_blk, n_kt, kvh;
  bool two;   // the second accumulator has rows
};
// units of CTA b: b, 2 n - 1 - b, 2 n + b, ... (n CTAs): with the longest first, every CTA's share is about the same
struct UnitIter {
  const PrefillArgs& a;
  int round = 0, kvh_ahead = 0;
  PrefillUnit ahead;   // the next unit, requested while the one before is worked on
  __device__ explicit UnitIter(const PrefillArgs& a_) : a(a_) { fetch(); }
  __device__ void fetch() {
    const int n = gridDim.x, i = round * n + ((round & 1) ? n - 1 - (int)blockIdx.x : (int)blockIdx.x);
    ahead.rows = 0;
    if (i >= a.n_units) return;   // the last round is the only one that is not full
    const int4 v = __ldg(reinterpret_cast<const int4*>(a.units) + i / a.n_kv);
    ahead = PrefillUnit{v.x, v.y, v.z, v.w};
    kvh_ahead = i % a.n_kv;
  }
  __device__ bool next(Unit& u) {
    if (ahead.rows == 0) return false;
    static_cast<PrefillUnit&>(u) = ahead;
    u.kvh = kvh_ahead;
    ++round;
    fetch();
    u.n_blk = (u.pos0 + u.rows - 1) / KV_BLOCK + 1;
    u.n_kt = (u.n_blk + PT_BLOCKS - 1) / PT_BLOCKS;
    u.two = u.rows > a.TM;
    return true;
  }
};

// dims 4 lane .. 4 lane + 3 of a token of a V block
__device__ __forceinline__ const __nv_bfloat16* value_of(const __nv_bfloat16* block, int token, int lane) {
  return block + token * HEAD_DIM + ((lane >> 1) ^ (token & 7)) * 8 + (lane & 1) * 4;
}
// One row by a warp, in the order of the keys: lane = token for the scores (twice), lane = four dims for the values, whose weights sum to
// one, so that no sum passes the largest value.
__device__ __forceinline__ void attend_row(const PrefillArgs& a, int block_row, int kvh, int head, int row, int pos) {
  const int lane = (int)lane_id();
  const float sl2 = a.minus != 0 ? -a.sl2 : a.sl2;
  const uint4* q = reinterpret_cast<const uint4*>(a.qkv + (size_t)row * a.qkv_ld + (size_t)head * HEAD_DIM);
  auto lo = [](uint32_t w) { return __uint_as_float(w << 16); };
  auto hi = [](uint32_t w) { return __uint_as_float(w & 0xffff0000u); };
  auto tile_of = [&](int b) { return ((size_t)a.block_table[(size_t)block_row * a.bt_stride + b] * a.n_kv + kvh) * (KV_BLOCK * HEAD_DIM); };
  auto score = [&](int b) {   // of the lane's token of block b
    if (b * KV_BLOCK + lane > pos) return -INFINITY;
    const __nv_bfloat16* from = a.k_cache + tile_of(b) + lane * 8;
    float s = 0.f;
#pragma unroll 2
    for (int c = 0; c < HEAD_DIM / 8; ++c) {
      const uint4 k = *reinterpret_cast<const uint4*>(from + c * (KV_BLOCK * 8)), x = q[c];
      s = fmaf(lo(x.x), lo(k.x), s); s = fmaf(hi(x.x), hi(k.x), s);
      s = fmaf(lo(x.y), lo(k.y), s); s = fmaf(hi(x.y), hi(k.y), s);
      s = fmaf(lo(x.z), lo(k.z), s); s = fmaf(hi(x.z), hi(k.z), s);
      s = fmaf(lo(x.w), lo(k.w), s); s = fmaf(hi(x.w), hi(k.w), s);
    }
    return s * sl2;
  };
  float m = -INFINITY, l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int b = 0; b <= pos / KV_BLOCK; ++b) {   // maximum and sum of the lane's tokens
    const float x = score(b), top = fmaxf(m, x);
    if (top > -INFINITY) l = l * ex2(m - top) + ex2(x - top);
    m = top;
  }
  float ref = m;
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) ref = fmaxf(ref, __shfl_xor_sync(0xffffffffu, ref, i));
  l *= ex2(m - ref);
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) l += __shfl_xor_sync(0xffffffffu, l, i);
  const float inv = 1.f / l;
#pragma unroll 1
  for (int b = 0; b <= pos / KV_BLOCK; ++b) {
    const float p = ex2(score(b) - ref) * inv;
    const int n = min(KV_BLOCK, pos - b * KV_BLOCK + 1);   // (hidden keys are not touched)
#pragma unroll 4
    for (int t = 0; t < n; ++t) {
      const float w = __shfl_sync(0xffffffffu, p, t);
      const uint2 v = *reinterpret_cast<const uint2*>(value_of(a.v_cache + tile_of(b), t, lane));
      o[0] = fmaf(w, lo(v.x), o[0]); o[1] = fmaf(w, hi(v.x), o[1]);
      o[2] = fmaf(w, lo(v.y), o[2]); o[3] = fmaf(w, hi(v.y), o[3]);
    }
  }
  *reinterpret_cast<uint2*>(a.out + (size_t)row * a.out_ld + (size_t)head * HEAD_DIM + lane * 4) = make_uint2(cvt2(o[0], o[1]), cvt2(o[2], o[3]));
}

// The CTA's rows that came out with numbers that are not finite, by its softmax warps, which have stored them all.  Where a key that the
// row sees accounts for them they stand: a unit's values are looked through once for the first such key of every dim, so that a
// sequence which has overflowed costs no more than that (a row summed again reads all of its keys twice, 32 loads in flight at most).
template <int ACC>
__device__ __noinline__ void sum_again(const PrefillArgs& a) {
  const int lane = (int)lane_id();
  auto odd = [](const uint2& w) {   // one bit per number of four
    const uint32_t e = 0x7f80u;
    return ((w.x & e) == e) | ((w.x >> 16 & e) == e) << 1 | ((w.y & e) == e) << 2 | ((w.y >> 16 & e) == e) << 3;
  };
  Unit u;
  for (UnitIter it(a); it.next(u);) {
    int first[4] = {-1, -1, -1, -1};   // of the lane's dims: the first key whose value is not finite (none: behind the last key)
    for (int r = threadIdx.x >> 5; r < u.rows * a.G; r += 4 * ACC) {
      const int t = r / a.G, row = u.row0 + t, head = u.kvh * a.G + r - t * a.G, pos = u.pos0 + t;
      const int mine = odd(*reinterpret_cast<const uint2*>(a.out + (size_t)row * a.out_ld + (size_t)head * HEAD_DIM + lane * 4));
      if (!__any_sync(0xffffffffu, mine != 0)) continue;
      if (first[0] < 0) {
        int seen = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) first[e] = u.n_blk * KV_BLOCK;
        for (int b = 0; b < u.n_blk && !__all_sync(0xffffffffu, seen == 15); ++b) {
          const int block = a.block_table[(size_t)u.block_row * a.bt_stride + b];
          const __nv_bfloat16* from = a.v_cache + ((size_t)block * a.n_kv + u.kvh) * (KV_BLOCK * HEAD_DIM);
#pragma unroll 4
          for (int k = 0; k < KV_BLOCK; ++k) {
            const int now = odd(*reinterpret_cast<const uint2*>(value_of(from, k, lane))) & ~seen;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (now >> e & 1) first[e] = b * KV_BLOCK + k;
            seen |= now;
          }
        }
      }
      int hidden = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) hidden |= (first[e] > pos) << e;
      if (__any_sync(0xffffffffu, (mine & hidden) != 0)) attend_row(a, u.block_row, u.kvh, head, row, pos);
    }
  }
}

template <int ACC, int BLOCKS>
__global__ void __launch_bounds__(PT_THREADS(ACC), BLOCKS == 1 ? 3 : 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap vmap, const __grid_constant__ PrefillArgs a) {
  constexpr int PT_WARP_COPY = 4 * ACC, PT_WARP_MMA = PT_WARP_COPY + 1, PT_STAGES = ACC;
  const int tile_blocks = ACC == 2 ? PT_BLOCKS : a.blocks, ring_bytes = tile_blocks * PT_BLOCK_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;
  uint8_t* k_s = q_s + ACC * PT_TILE_BYTES;
  uint8_t* v_s = k_s + PT_STAGES * ring_bytes;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(v_s + PT_STAGES * ring_bytes);
  uint64_t* q_empty = q_full + 1;
  uint64_t* k_full = q_empty + 1;
  uint64_t* k_empty = k_full + PT_STAGES;
  uint64_t* v_full = k_empty + PT_STAGES;
  uint64_t* v_empty = v_full + PT_STAGES;
  uint64_t* s_full = v_empty + PT_STAGES;   // [2]
  uint64_t* p_full = s_full + 2;            // [2]
  uint64_t* o_full = p_full + 2;            // [2]
  uint32_t* tmem_base_smem = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_base_smem + 1);
  volatile int* redo = gave_up + 1;         // rows of the CTA have to be summed again

  const int warp = threadIdx.x >> 5, lane = (int)lane_id();
  // units and block table are written by the host before the step: they are read while the kernel before this one still runs
  UnitIter it(a);
  auto tiles = [](const Unit& u) { return ACC == 2 ? u.n_kt : 1; };
  if (warp == PT_WARP_MMA) {
    if (elect_one()) {
      mbar_init(q_full, 1);
      mbar_init(q_empty, 1);
      for (int i = 0; i < PT_STAGES; ++i) {
        mbar_init(&k_full[i], 1);
        mbar_init(&k_empty[i], 1);
        mbar_init(&v_full[i], 1);
        mbar_init(&v_empty[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&s_full[i], 1);
        mbar_init(&p_full[i], 4);
        mbar_init(&o_full[i], 1);
      }
      *gave_up = 0;
      *redo = 0;
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc<256 * ACC>(tmem_base_smem);
  }
  if (warp == PT_WARP_COPY && lane == 0) {
    tma_prefetch_desc(&qmap);
    tma_prefetch_desc(&vmap);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_smem;   // [S0 | S1 | O0 | O1] or [S0 | O0], 128 columns each
  griddep_launch();
  Unit u;
  bool ok = true;
  if (warp >= PT_WARP_COPY) {
    if constexpr (ACC == 2) set_regs<PT_REGS_OTHER, false>();
    if (warp == PT_WARP_COPY) {
      // ===================== copies =====================
      int kst = 0, vst = 0;
      uint32_t kph = 1, vph = 1, qph = 1;   // the first pass over a ring finds it empty
      const uint32_t q_bytes = 2u * 64 * 2 * (uint32_t)(a.G * a.TM);
      bool have = it.next(u);
      auto block_of = [&](int j) {   // this lane's block of tile j
        const int b = j * PT_BLOCKS + lane;
        return lane < PT_BLOCKS && b < u.n_blk ? a.block_table[(size_t)u.block_row * a.bt_stride + b] : 0;
      };
      int blk = have ? block_of(0) : 0;
      griddep_wait();   // q, K and V
      for (; ok && have; have = it.next(u), blk = have ? block_of(0) : 0) {
        ok = __all_sync(0xffffffffu, bounded_wait(q_empty, qph, a.err));
        if (!ok) break;
        qph ^= 1;
        if (lane == 0) {
          mbar_arrive_expect_tx(q_full, u.two ? 2 * q_bytes : q_bytes);
          for (int g = 0; g < (u.two ? 2 : 1); ++g)
            for (int h = 0; h < 2; ++h)
              tma_load_3d(&qmap, q_full, q_s + g * PT_TILE_BYTES + h * (PT_TILE_BYTES / 2), h * 64, u.kvh * a.G, u.row0 + g * a.TM);
        }
        for (int j = 0; j < tiles(u); ++j) {
          const int nb = min(PT_BLOCKS, u.n_blk - j * PT_BLOCKS);
          ok = __all_sync(0xffffffffu, bounded_wait(&k_empty[kst], kph, a.err));
          if (!ok) break;
          if (lane == 0) mbar_arrive_expect_tx(&k_full[kst], nb * PT_BLOCK_BYTES);
          __syncwarp();
          // a block by itself lies as in the cache (one copy; sixteen take the copy unit half a microsecond)
          if (nb == 1 && lane == 0)
            bulk_load_1d(k_s + kst * ring_bytes, a.k_cache + ((size_t)blk * a.n_kv + u.kvh) * (KV_BLOCK * HEAD_DIM), PT_BLOCK_BYTES, &k_full[kst]);
          for (int b = lane >> 4; nb > 1 && b < PT_BLOCKS; b += 2) {   // lane -> (block, chunk)
            const int pb = __shfl_sync(0xffffffffu, blk, b);
            const int c = lane & 15;
            if (b < nb)
              bulk_load_1d(k_s + kst * ring_bytes + c * (tile_blocks * KV_BLOCK * 16) + b * (KV_BLOCK * 16),
                           a.k_cache + ((size_t)pb * a.n_kv + u.kvh) * (KV_BLOCK * HEAD_DIM) + c * (KV_BLOCK * 8), KV_BLOCK * 16, &k_full[kst]);
          }
          if (++kst == PT_STAGES) kst = 0, kph ^= 1;
          ok = __all_sync(0xffffffffu, bounded_wait(&v_empty[vst], vph, a.err));
          if (!ok) break;
          if (lane == 0) mbar_arrive_expect_tx(&v_full[vst], nb * PT_BLOCK_BYTES);
          __syncwarp();
          if (lane < nb)
            tma_load_3d(&vmap, &v_full[vst], v_s + vst * ring_bytes + lane * PT_BLOCK_BYTES, 0, (blk * a.n_kv + u.kvh) * KV_BLOCK, 0);
          if (++vst == PT_STAGES) vst = 0, vph ^= 1;
          blk = block_of(j + 1);
        }
      }
    } else if (warp == PT_WARP_MMA) {
      // ===================== MMAs =====================
      int kst = 0, vst = 0;
      uint32_t kph = 0, vph = 0, qph = 0, pph[2] = {0, 0};
      // O += P V for the blocks of a tile; both operands' 16 tokens of a step at a time
      const uint32_t idesc_pv = make_idesc_bf16(128, HEAD_DIM) | (1u << 16);   // B (V) has its dims contiguous
      auto scores = [&](int g, int nb) {
        const uint32_t idesc = make_idesc_bf16(128, nb * KV_BLOCK) | a.minus;
        const uint32_t q = smem_u32(q_s + g * PT_TILE_BYTES), k = smem_u32(k_s + kst * ring_bytes);
        const uint32_t chunk = (nb == 1 ? 1 : tile_blocks) * KV_BLOCK * 16;
#pragma unroll
        for (int ks = 0; ks < HEAD_DIM / 16; ++ks)
          tc_mma_f16(tmem_base + g * 128, make_smem_desc_sw128(q + ((7 - ks) >> 2) * (PT_TILE_BYTES / 2) + ((7 - ks) & 3) * 32),
                     smem_desc(k + (7 - ks) * 2 * chunk, chunk, 128, 0), idesc, ks > 0);
        tc_commit(&s_full[g]);
      };
      auto values = [&](int g, int nb, bool first) {
        const uint32_t v = smem_u32(v_s + vst * ring_bytes);
        for (int ks = 0; ks < 2 * nb; ++ks) {
          const uint64_t vd = smem_desc(v + (ks >> 1) * PT_BLOCK_BYTES + (ks & 1) * 2048, PT_BLOCK_BYTES / 2, 1024, 2);
          mma_ts(tmem_base + ACC * 128 + g * 128, tmem_base + g * 128 + ks * 8, vd, idesc_pv, !(first && ks == 0));
          mma_ts(tmem_base + ACC * 128 + g * 128, tmem_base + g * 128 + 64 + ks * 8, vd, idesc_pv, 1);
        }
      };
      while (ok && it.next(u)) {
        const int groups = ACC == 2 && u.two ? 2 : 1;
        auto blocks = [&](int j) { return min(PT_BLOCKS, u.n_blk - j * PT_BLOCKS); };
        ok = __all_sync(0xffffffffu, bounded_wait(q_full, qph, a.err) && bounded_wait(&k_full[kst], kph, a.err));
        if (!ok) break;
        qph ^= 1;
        tc_fence_after();
        if (elect_one()) {
          for (int g = 0; g < groups; ++g) scores(g, blocks(0));
          tc_commit(&k_empty[kst]);
          if (tiles(u) == 1) tc_commit(q_empty);
        }
        __syncwarp();
        if (++kst == PT_STAGES) kst = 0, kph ^= 1;
        for (int j = 0; j < tiles(u) && ok; ++j) {
          const bool more = j + 1 < tiles(u);
          ok = __all_sync(0xffffffffu, bounded_wait(&v_full[vst], vph, a.err));
          for (int g = 0; g < groups && ok; ++g) {
            ok = __all_sync(0xffffffffu, bounded_wait(&p_full[g], pph[g], a.err) && (g > 0 || !more || bounded_wait(&k_full[kst], kph, a.err)));
            if (!ok) break;
            pph[g] ^= 1;
            tc_fence_after();
            if (elect_one()) {
              const bool last = g == groups - 1;
              values(g, blocks(j), j == 0);
              if (more) scores(g, blocks(j + 1));
              if (last) {
                tc_commit(&v_empty[vst]);
                if (more) tc_commit(&k_empty[kst]);
                if (j + 2 == tiles(u)) tc_commit(q_empty);
              }
              if (!more) tc_commit(&o_full[g]);
            }
            __syncwarp();
          }
          if (++vst == PT_STAGES) vst = 0, vph ^= 1;
          if (more && ++kst == PT_STAGES) kst = 0, kph ^= 1;
        }
      }
    }
  } else {
    // ===================== softmax: thread = row =====================
    if constexpr (ACC == 2) set_regs<PT_REGS_SOFTMAX, true>();
    const int g = warp >> 2;
    const int r = (warp & 3) * 32 + lane, tok = r / a.G, head = r - tok * a.G;
    const int tok_lo = (warp & 3) * 32 / a.G;                       // first token of the warp
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_t = tmem_base + g * 128 + lanes, o_t = tmem_base + ACC * 128 + g * 128 + lanes;
    const uint64_t sl2_2 = pack2(a.sl2, a.sl2), minus1 = pack2(-1.f, -1.f);
    uint32_t sph = 0, oph = 0;
    griddep_wait();   // `out` may still be read
    while (ok && it.next(u)) {
      if (g == 1 && !u.two) continue;
      const int pos = u.pos0 + g * a.TM + tok, pos_lo = u.pos0 + g * a.TM + tok_lo;
      float m = 0.f, l = 0.f;
      for (int j = 0; j < tiles(u); ++j) {
        const int nb = BLOCKS == 1 ? 1 : min(PT_BLOCKS, u.n_blk - j * PT_BLOCKS);
        const int lim = pos - j * PT_KV;   // last column this row sees
        const bool mask = j * PT_KV + nb * KV_BLOCK - 1 > pos_lo;
        ok = __all_sync(0xffffffffu, bounded_wait(&s_full[g], sph, a.err));
        if (!ok) break;
        sph ^= 1;
        tc_fence_after();
        uint32_t s[BLOCKS * KV_BLOCK];
        // (one way out of each loop: a prompt of a block would else run past all of their code, which no cache holds yet)
#pragma unroll
        for (int c = 0; c < BLOCKS; ++c) {
          if (c >= nb) break;
          tmem_ld_x32(s_t + c * 32, s + c * 32);
        }
        tmem_ld_wait();
        if (mask) {
#pragma unroll
          for (int c = 0; c < BLOCKS; ++c) {
            if (c >= nb) break;
#pragma unroll
            for (int i = c * 32; i < c * 32 + 32; ++i)
              if (i > lim) s[i] = __float_as_uint(-INFINITY);
          }
        }
        float mx[PT_BLOCKS] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < BLOCKS; ++c) {
          if (c >= nb) break;
#pragma unroll
          for (int i = 0; i < 32; i += 2) mx[c] = fmaxf(mx[c], fmaxf(__uint_as_float(s[c * 32 + i]), __uint_as_float(s[c * 32 + i + 1])));
        }
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.sl2;
        if (j == 0) {
          m = top;
        } else if (__any_sync(0xffffffffu, top > m + PT_SLACK)) {
          // the products that wrote O retired before these scores did
          const float f = top > m + PT_SLACK ? ex2(m - top) : 1.f;
          if (top > m + PT_SLACK) m = top;
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
        for (int c = 0; c < 2 * BLOCKS; ++c) {
          if (c >= 2 * nb) break;
          uint32_t hi[8], lo[8];
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
            hi[i] = cvt2(x, y);
            const uint64_t back = pack2(__uint_as_float(hi[i] << 16), __uint_as_float(hi[i] & 0xffff0000u));
            unpack2(fma2(back, minus1, p), x, y);
            lo[i] = cvt2(x, y);
          }
          tmem_st_x8(s_t + c * 8, hi);
          tmem_st_x8(s_t + 64 + c * 8, lo);
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
      const float inv = 1.f / l;
      const bool wanted = tok < a.TM && g * a.TM + tok < u.rows;
      __nv_bfloat16* dst = a.out + (size_t)(u.row0 + g * a.TM + tok) * a.out_ld + (size_t)(u.kvh * a.G + head) * HEAD_DIM;
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
  if (*redo != 0 && *gave_up == 0 && warp < PT_WARP_COPY) sum_again<ACC>(a);
  // after a wait that ran out copies and MMAs of the other roles may be in flight; they are done long before this millisecond is over
  if (*gave_up)
    for (const long long t0 = clock64(); clock64() - t0 < 2000000ll;) {}
  __syncthreads();
  if (warp == PT_WARP_MMA) {
    tc_fence_after();
    tmem_dealloc<256 * ACC>(tmem_base);
  }
}

template <int ACC, int BLOCKS>
cudaError_t launch(const CUtensorMap& qm, const CUtensorMap& vm, const PrefillArgs& a, int num_sms, cudaStream_t stream) {
  static const cudaError_t attr = cudaFuncSetAttribute(attn_prefill_kernel<ACC, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PT_SMEM(ACC, BLOCKS));
  if (attr != cudaSuccess) return attr;
  return launch_k(attn_prefill_kernel<ACC, BLOCKS>, dim3(std::min(a.n_units, num_sms)), dim3(PT_THREADS(ACC)), PT_SMEM(ACC, ACC == 2 ? BLOCKS : a.blocks), stream,
                  qm, vm, a);
}

int accumulator_tokens(int G) { return std::max(128 / G & ~7, 8); }

}  // namespace

// Units of the prompts and portions among `seqs` (q_len > 1), those with the most cache tiles first (ties in order).  Where no sequence
// has more than one tile of keys and the SMs take all units at once, a unit is one accumulator's rows and the launch the small one:
// *short_blocks is then the number of cache blocks of the longest sequence, else 0.
int prefill_units_build(PrefillUnit* units, const AttnSeq* seqs, int n_seqs, int G, int n_kv, int num_sms, int* short_blocks) {
  const int rows = accumulator_tokens(G);
  int keys = 0;
  long long pieces = 0;
  for (int s = 0; s < n_seqs; ++s)
    if (seqs[s].q_len > 1) keys = std::max(keys, seqs[s].kv_len), pieces += (seqs[s].q_len + rows - 1) / rows;
  *short_blocks = keys <= PT_KV && pieces * n_kv <= num_sms ? (keys + KV_BLOCK - 1) / KV_BLOCK : 0;
  const int step = *short_blocks > 0 ? rows : 2 * rows;
  int n = 0;
  for (int s = 0; s < n_seqs; ++s) {
    const AttnSeq& q = seqs[s];
    if (q.q_len <= 1) continue;
    for (int q0 = 0; q0 < q.q_len; q0 += step)
      units[n++] = PrefillUnit{q.q_start + q0, std::min(step, q.q_len - q0), q.kv_len - q.q_len + q0, q.block_row};
  }
  std::stable_sort(units, units + n, [](const PrefillUnit& x, const PrefillUnit& y) {
    return (x.pos0 + x.rows - 1) / PT_KV > (y.pos0 + y.rows - 1) / PT_KV;
  });
  return n;
}

cudaError_t attn_prefill_launch(const __nv_bfloat16* qkv, int qkv_ld, const __nv_bfloat16* k_cache, const __nv_bfloat16* v_cache, int n_blocks,
                                const PrefillUnit* units, int n_units, int short_blocks, const int32_t* block_table, int bt_stride,
                                __nv_bfloat16* out, int out_ld, int T, int n_q, int n_kv, float scale, int num_sms, cudaStream_t stream) {
  if (n_units <= 0) return cudaSuccess;
  if (n_kv <= 0 || n_q % n_kv != 0) return cudaErrorInvalidValue;
  const int G = n_q / n_kv;
  if (G > 8) return cudaErrorInvalidValue;
  PrefillArgs a{};
  cudaError_t e = gemm_pair_word(&a.err);
  if (e != cudaSuccess) return e;
  a.qkv = qkv; a.k_cache = k_cache; a.v_cache = v_cache; a.units = units; a.block_table = block_table;
  a.out = out;
  a.n_units = n_units * n_kv; a.bt_stride = bt_stride; a.qkv_ld = qkv_ld; a.out_ld = out_ld; a.n_kv = n_kv; a.G = G; a.TM = accumulator_tokens(G);
  a.sl2 = scale != 0.f ? fabsf(scale) * 1.4426950408889634f : 1e-30f;   // hidden scores are -inf before they are scaled
  a.minus = scale < 0.f ? 1u << 13 : 0u;
  CUtensorMap qm, vm;
  // q: (dim, head, token), boxes of 64 dims x G heads x TM tokens; v: (64 dims, cache row, half of the dims)
  if (make_tmap_bf16_3d(&qm, qkv, {(uint64_t)HEAD_DIM, (uint64_t)n_q, (uint64_t)T}, {HEAD_DIM * 2ull, (uint64_t)qkv_ld * 2},
                        {64, (uint32_t)G, (uint32_t)a.TM}, true) != 0 ||
      make_tmap_bf16_3d(&vm, v_cache, {64, (uint64_t)n_blocks * n_kv * KV_BLOCK, 2}, {HEAD_DIM * 2ull, 128}, {64, KV_BLOCK, 2}, false) != 0)
    return cudaErrorInvalidValue;
  a.blocks = short_blocks;
  if (short_blocks == 1) return launch<1, 1>(qm, vm, a, num_sms, stream);
  return short_blocks > 0 ? launch<1, PT_BLOCKS>(qm, vm, a, num_sms, stream) : launch<2, PT_BLOCKS>(qm, vm, a, num_sms, stream);
}

}  // namespace tgis
