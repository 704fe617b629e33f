// Causal flash attention for sm_100a: S = Q K^T and O += P V on tcgen05 tensor cores with the
// accumulators in tensor memory, operands staged by TMA, softmax in registers (one query row per
// thread, read from tensor memory with tcgen05.ld).  It stands in for the fused attention the
// reference gets from F.scaled_dot_product_attention (models/gpt_model.py:90-92).
//
// All three large kernels (forward, dQ, dK / dV) are persistent, one CTA per SM, and work on tiles of 128 queries by 128
// keys: one warp issues the TMA loads, one elected lane of a warp each stream of MMAs, and eight or sixteen warps do the
// softmax with S, dP (fp32), P and dS (bf16) in tensor memory.  What bounds them is the special function unit (16 exponentials per
// cycle and SM: 1024 cycles per pair of tiles) and, at D = 128, the tensor core (2048 cycles in dK / dV); what costs time on
// top are the waits between the roles, 200 to 300 cycles from an arrival to what it sets off.  So every product is issued as early
// as its operands allow, and nothing waits for a buffer that could be another one.
//   64 x 1024 x 12 heads of 64 (us, this against 128 x 64 tiles with two CTAs per SM): forward 183 / 250, dQ 237 / 368,
//   dK and dV 261 / 579; 32 heads of 128 with 8 kv heads at T = 4096: 133 / 170, 165 / 301, 250 / 473.
// Layouts: q [B*T, H*D], k / v [B*T, Hkv*D], out [B*T, H*D] (bf16, row-major), lse [B, H, T] fp32.
// Every mbarrier wait is bounded; a wait that gives up sets the status word and the CTA drains.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <atomic>
#include <mutex>
#include <type_traits>

#include "gemm.h"
#include "kernels.h"
#include "pdl.cuh"
#include "per_device.h"
#include "umma.cuh"

namespace dion {

namespace {

constexpr int kBM = 128;  // rows of a tile, of queries and of keys
constexpr float kRescaleThreshold = 8.f;  // log2 units

__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const float (&v)[32]) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The MMA-issuing thread is on the critical path of every kv iteration (tiles are small, so one
// tcgen05.mma runs for only 30-70 cycles); descriptors are therefore kept as two 32-bit halves and
// stepped with a single integer add: the start-address field (bits [0,14), units of 16 bytes) never
// carries because shared-memory offsets stay below 256 KB.
struct DescHalves {
  uint32_t lo, hi;
};
__device__ __forceinline__ DescHalves desc_halves(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  const uint64_t d = make_smem_desc(smem_addr, lbo_bytes, sbo_bytes);
  return DescHalves{(uint32_t)d, (uint32_t)(d >> 32)};
}
// D[tmem] (+)= A[smem] * B[smem], bf16, descriptors given as halves plus byte offsets
__device__ __forceinline__ void umma_ss_h(uint32_t tmem_d, DescHalves a, uint32_t a_off, DescHalves b, uint32_t b_off,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(tmem_d),
      "r"(a.lo + (a_off >> 4)), "r"(a.hi), "r"(b.lo + (b_off >> 4)), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts_h(uint32_t tmem_d, uint32_t tmem_a, DescHalves b, uint32_t b_off,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b.lo + (b_off >> 4)), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 operations in one instruction.  The softmax loops issue 7 to 14 instructions per score without them and are
// what the tensor core waits for; with them 3 to 5, of which one is the exponential.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  const __nv_bfloat162 h2 = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h2);
}

// untiled bulk copy global -> shared (both 16-byte aligned, size a multiple of 16), completing on `bar`
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem_dst)),
               "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// n / d for 0 <= n < 2^31 by a multiplication (Granlund and Montgomery, 1994); the integer division of the device takes some
// hundred cycles, and a role does several of them before it can start on a tile
struct FastDiv {
  uint32_t d, m, s;
  FastDiv() = default;
  explicit FastDiv(int divisor) : d((uint32_t)divisor), m(0), s(0) {
    while (s < 31 && (1u << s) < d) ++s;
    m = (uint32_t)(((1ull << 32) * ((1ull << s) - d)) / d + 1);
  }
  __device__ __forceinline__ int operator()(int n) const { return (int)((__umulhi((uint32_t)n, m) + (uint32_t)n) >> s); }
};

// What a persistent CTA works through: (sequence and head, tile) pairs, tile `level` 0 being the one with the most work.
// The pairs are taken in groups of as many heads as there are CTAs: a CTA then runs all tiles of one head, so every CTA
// does the same work per group and what it reads again is still in L2.  The heads that are left over are dealt out tile
// by tile, heaviest first, back and forth over the CTAs.
struct WorkPlan {  // made on the host
  int levels, whole, first, rem, total;  // tiles per head; rounds with a head for every CTA; the heads after them, their pairs
  FastDiv by_rem;
  WorkPlan() = default;
  WorkPlan(int levels_, int heads, int ctas)
      : levels(levels_), whole(heads / ctas * levels_), first(heads / ctas * ctas), rem(heads % ctas), total(rem * levels_),
        by_rem(rem > 0 ? rem : 1) {}
};
struct WorkList {
  const WorkPlan& plan;
  int head, level;  // the current pair
  int round = 0;
  bool valid = true;
  __device__ __forceinline__ explicit WorkList(const WorkPlan& p) : plan(p), head((int)blockIdx.x), level(0) {
    if (plan.whole == 0) leftover();
  }
  __device__ __forceinline__ void next() {
    ++round;
    if (round < plan.whole) {
      if (++level == plan.levels) {
        level = 0;
        head += (int)gridDim.x;
      }
    } else {
      leftover();
    }
  }
  __device__ __forceinline__ void leftover() {
    const int g = (int)gridDim.x, c = (int)blockIdx.x;
    const int r = round - plan.whole;
    const int k = r * g + ((r & 1) ? g - 1 - c : c);
    valid = k < plan.total;
    level = plan.by_rem(k);
    head = plan.first + (k - level * plan.rem);
  }
};

// Position in a ring of N stages and the parity of the barrier phase that fills it next
template <int N>
struct Ring {
  int s = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next() {
    if (++s == N) {
      s = 0;
      ph ^= 1u;
    }
  }
};

// 16 lanes x 32 fp32 columns: lane t receives, for k = 0..3, columns 8k + 2 (t & 3) and + 1 of row t >> 2 (v[4k], v[4k + 1])
// and of row (t >> 2) + 8 (v[4k + 2], v[4k + 3])
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// 128 rows x 32 bytes from shared memory (a K-major operand tile) to 8 columns of tensor memory
__device__ __forceinline__ void tmem_cp_128x32b(uint32_t taddr, DescHalves d, uint32_t off) {
  asm volatile("{\n\t.reg .b64 d;\n\tmov.b64 d, {%1, %2};\n\ttcgen05.cp.cta_group::1.128x256b [%0], d;\n\t}" ::"r"(taddr),
               "r"(d.lo + (off >> 4)), "r"(d.hi)
               : "memory");
}
// v[k] of lane q of each group of four becomes v[q] of lane k
__device__ __forceinline__ void quad_transpose(uint32_t (&v)[4], int lane) {
#pragma unroll
  for (int b = 1; b <= 2; b <<= 1) {
    const bool up = lane & b;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i & b) continue;
      const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i | b], b);
      if (up) v[i] = got;
      else v[i | b] = got;
    }
  }
}
// 32 accumulator rows (lane quadrant `quad`, COLS fp32 columns from `taddr`) to `out` as bf16, row r at out + (quad * 32 + r) *
// pitch, rows from `rows` on left out; kScaled: times the factor that the lane of the row holds.  Eight rows of 64 bytes per
// store instruction: with a row per lane each one touches 32 lines, and the stores of dV and dK took 3000 cycles per kv tile.
template <int COLS, bool kScaled = false>
__device__ __forceinline__ void store_rows(uint32_t taddr, int quad, int lane, __nv_bfloat16* out, long long pitch, int rows,
                                           float scale_of_lane = 1.f) {
#pragma unroll
  for (int c0 = 0; c0 < COLS; c0 += 64) {  // all loads of 64 columns first: they take as long as one
    constexpr int CH = COLS < 64 ? COLS / 32 : 2;
    float v[2][CH][16];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
#pragma unroll
      for (int c = 0; c < CH; ++c)
        tmem_ld_16x256b_x4(taddr + ((uint32_t)(quad * 32 + hh * 16) << 16) + c0 + c * 32, v[hh][c]);
    tmem_ld_wait();
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int row = quad * 32 + hh * 16 + (lane >> 2);
      __nv_bfloat16* dst = out + row * pitch + c0 + (lane & 3) * 8;
      float f0 = 1.f, f1 = 1.f;  // of this lane's two rows
      if constexpr (kScaled) {
        f0 = __shfl_sync(0xffffffffu, scale_of_lane, hh * 16 + (lane >> 2));
        f1 = __shfl_sync(0xffffffffu, scale_of_lane, hh * 16 + 8 + (lane >> 2));
      }
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float* w = &v[hh][c][4 * k];
          lo[k] = kScaled ? pack_bf16x2(w[0] * f0, w[1] * f0) : pack_bf16x2(w[0], w[1]);
          hi[k] = kScaled ? pack_bf16x2(w[2] * f1, w[3] * f1) : pack_bf16x2(w[2], w[3]);
        }
        quad_transpose(lo, lane);
        quad_transpose(hi, lane);
        if (row < rows) *reinterpret_cast<uint4*>(dst + c * 32) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        if (row + 8 < rows) *reinterpret_cast<uint4*>(dst + 8 * pitch + c * 32) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      }
    }
  }
}

// D[128 x 128] = A B^T over the head dimension, both K-major tiles; A from tensor memory (a_col) where kTmemA
template <int D, bool kTmemA>
__device__ __forceinline__ void scores(uint32_t d_col, DescHalves a, uint32_t a_col, DescHalves b, uint32_t b_off) {
  constexpr uint32_t idesc = make_instr_desc(1, kMajorK, kMajorK, kBM, kBM);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const uint32_t off = (kk >> 2) * (kBM * 128) + (kk & 3) * 32;
    if constexpr (kTmemA) umma_ts_h(d_col, a_col + kk * 8, b, b_off + off, idesc, kk > 0 ? 1u : 0u);
    else umma_ss_h(d_col, a, off, b, b_off + off, idesc, kk > 0 ? 1u : 0u);
  }
}
// a K-major tile of 128 rows into tensor memory as the A operand of `scores`
template <int D>
__device__ __forceinline__ void keep_tile(uint32_t col, DescHalves a) {
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) tmem_cp_128x32b(col + kk * 8, a, (kk >> 2) * (kBM * 128) + (kk & 3) * 32);
}

// ---------------------------------------------------------------------------------- forward
struct AttnParams {
  __nv_bfloat16* out;
  float* lse;
  int B, T, H, Hkv;
  float scale_log2;  // softmax scale * log2(e)
  int pair;          // query tiles per work item: 2, or 1 where there are SMs to spare
  WorkPlan plan;
  FastDiv by_heads, by_group;
  int* status;
};


// Register shares of the first warpgroup and of the eight softmax warps after it: together no more than the 384 x 168 that
// the launch has, or the larger share waits forever
template <int kFirst, int kSoftmax>
__device__ __forceinline__ void give_registers() {
  static_assert(128 * kFirst + 256 * kSoftmax <= 384 * 168 && kFirst % 8 == 0 && kSoftmax % 8 == 0);
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFirst));
}
template <int kFirst, int kSoftmax>
__device__ __forceinline__ void take_registers() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmax));
}
constexpr int kFwdThreads = 32 * 12;  // TMA; products of either query tile; a spare; four softmax warps per query tile

template <int D>
struct AttnCfg {
  static constexpr int PANELS = D / 64;             // 128-byte panels along the head dimension
  static constexpr int TILE_BYTES = kBM * D * 2;    // 128 rows of Q, K or V
  static constexpr int K_STAGES = D == 128 ? 3 : 4, V_STAGES = D == 128 ? 2 : 4;
  static constexpr int SMEM = (2 + K_STAGES + V_STAGES) * TILE_BYTES + 256;
  // tensor memory: S and O of both query tiles; D = 64 has room for P beside S, D = 128 writes P over S
  static constexpr bool P_APART = D == 64;
  static constexpr int S_COL = 0;                   // + 128 per query tile
  static constexpr int O_COL = 2 * kBM;             // + D
  static constexpr int P_COL = P_APART ? 2 * kBM + 2 * D : S_COL;
  static constexpr int P_TILE = P_APART ? 64 : kBM;  // columns from one query tile's P to the other's
  static constexpr int TMEM_COLS = 512;
  static_assert(P_COL + 2 * 64 <= TMEM_COLS && O_COL + 2 * D <= TMEM_COLS && SMEM <= 232448, "one CTA per SM");
};

// One CTA per SM runs through pairs of query tiles; both share the K and V tiles, each has four softmax warps with one
// query row per thread.  While one pair of warps per scheduler takes exponentials (1024 cycles of the special function
// unit per tile, what bounds the kernel at D = 64), the other tile's row maximum, stores and products run.  At D = 64 the
// next S of a tile is multiplied as soon as this one is in registers.
template <int D>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const AttnParams p) {
  using C = AttnCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                                  // two tiles
  uint8_t* sK = sQ + 2 * C::TILE_BYTES;
  uint8_t* sV = sK + C::K_STAGES * C::TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + C::V_STAGES * C::TILE_BYTES);
  uint64_t* q_full = bars;       // one per query tile, as the next five
  uint64_t* q_empty = bars + 2;
  uint64_t* s_full = bars + 4;
  uint64_t* s_free = bars + 6;   // four warps: S is in registers (P_APART)
  uint64_t* p_full = bars + 8;   // four warps
  uint64_t* pv_done = bars + 10;  // O += P V retired: O stable, P free
  uint64_t* k_full = bars + 12;  // K_STAGES each
  uint64_t* k_empty = k_full + C::K_STAGES;
  uint64_t* v_full = k_empty + C::K_STAGES;  // V_STAGES each
  uint64_t* v_empty = v_full + C::V_STAGES;
  uint64_t* bars_end = v_empty + C::V_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_end);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = (int)warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int tiles = (p.T + kBM - 1) / kBM;
  const int items = (tiles + p.pair - 1) / p.pair;  // per head
  WorkList work(p.plan);                            // level 0 = the last query tiles, which see all kv tiles
  if (smem_u32(smem) & 1023) {                      // the 128-byte swizzle repeats every 1024 bytes
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, kStatusBadArgument);
    return;
  }

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    for (uint64_t* b = bars; b < bars_end; ++b)
      mbar_init(b, (b >= s_free && b < pv_done) ? 4 : ((b >= k_empty && b < v_full) || b >= v_empty) ? 2 : 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  pdl_trigger();
  pdl_wait();
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  if (warp < 4) {
    give_registers<96, 200>();
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      if (lane == 0) {
        bool ok = true;
        Ring<C::K_STAGES> ks;
        Ring<C::V_STAGES> vs;
        int nq[2] = {0, 0};  // loads of each query tile's buffer
        auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col, int row, int seq) {
#pragma unroll
          for (int c = 0; c < C::PANELS; ++c) tma_load_3d(dst + c * (kBM * 128), map, bar, col + c * 64, row, seq);
        };
        for (; ok && work.valid; work.next()) {
          const int q0 = (items - 1 - work.level) * p.pair, q1 = min(q0 + p.pair, tiles);
          const int b = p.by_heads(work.head), h = work.head - b * p.H, hk = p.by_group(h);
          for (int j = 0; j < q1 && ok; ++j) {
            if (j == 0) {
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                if (q0 + x >= q1) continue;
                ok = ok && mbar_wait(&q_empty[x], (nq[x] & 1) ^ 1u, abort_flag);
                if (!ok) break;
                mbar_arrive_expect_tx(&q_full[x], C::TILE_BYTES);
                load(sQ + x * C::TILE_BYTES, &tmap_q, &q_full[x], h * D, (q0 + x) * kBM, b);
                ++nq[x];
              }
              if (!ok) break;
            }
            ok = mbar_wait(&k_empty[ks.s], ks.ph ^ 1u, abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(&k_full[ks.s], C::TILE_BYTES);
            load(sK + ks.s * C::TILE_BYTES, &tmap_k, &k_full[ks.s], hk * D, j * kBM, b);
            ok = mbar_wait(&v_empty[vs.s], vs.ph ^ 1u, abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(&v_full[vs.s], C::TILE_BYTES);
            load(sV + vs.s * C::TILE_BYTES, &tmap_v, &v_full[vs.s], hk * D, j * kBM, b);
            ks.next();
            vs.next();
          }
        }
        if (!ok) {
          *abort_flag = 1;
          if (p.status) atomicCAS(p.status, 0, kStatusProducerTimeout);
        }
      }
    } else if (warp < 3) {
      // ---------------------------------------------------------------- S = Q K^T and O += P V of one query tile
      // Each tile has an issuing warp of its own: with one for both, a tile that is ahead waits for the other's softmax.
      if (elect_one()) {
        const int x = warp - 1;
        constexpr uint32_t idesc = make_instr_desc(1, kMajorK, kMajorMN, kBM, D);
        const DescHalves dq_ = desc_halves(smem_u32(sQ) + x * C::TILE_BYTES, 16, 1024), dk_ = desc_halves(smem_u32(sK), 16, 1024);
        const DescHalves dv_ = desc_halves(smem_u32(sV), kBM * 128, 1024);
        const uint32_t s_col = tmem_base + C::S_COL + x * kBM, p_col = tmem_base + C::P_COL + x * C::P_TILE;
        const uint32_t o_col = tmem_base + C::O_COL + x * D;
        bool ok = true;
        Ring<C::K_STAGES> ks;
        Ring<C::V_STAGES> vs;
        uint32_t ph = 0;    // of the tile whose P is awaited
        uint32_t nq = 0;    // query tiles so far
        // S of kv tile j of the item that `w` stands at; `last` is the tile's last one
        auto issue_s = [&](int j, int last) {
          ok = ok && mbar_wait(&k_full[ks.s], ks.ph, abort_flag) && (j > 0 || mbar_wait(&q_full[x], nq & 1, abort_flag));
          if (!ok) return;
          tc_fence_after();
          scores<D, false>(s_col, dq_, 0, dk_, ks.s * C::TILE_BYTES);
          umma_commit(&s_full[x]);
          umma_commit(&k_empty[ks.s]);
          if (j == last) {
            umma_commit(&q_empty[x]);
            ++nq;
          }
          ks.next();
        };
        // a pair of K and V tiles that this query tile does not see: passed on once it has arrived
        auto skip = [&]() {
          ok = ok && mbar_wait(&k_full[ks.s], ks.ph, abort_flag);
          if (ok) mbar_arrive(&k_empty[ks.s]);
          ok = ok && mbar_wait(&v_full[vs.s], vs.ph, abort_flag);
          if (ok) mbar_arrive(&v_empty[vs.s]);
          ks.next();
          vs.next();
        };
        auto last_of = [&](const WorkList& w) {  // this tile's last kv tile; -1: the item has no such tile
          const int qt = (items - 1 - w.level) * p.pair + x;
          return x < p.pair && qt < tiles ? qt : -1;
        };
        int last = last_of(work);
        if (last >= 0) issue_s(0, last);
        while (ok && work.valid) {
          const int q1 = min((items - 1 - work.level) * p.pair + p.pair, tiles);
          for (int j = 0; j <= last && ok; ++j) {
            if (C::P_APART && j < last) {
              ok = mbar_wait(&s_free[x], ph, abort_flag);
              issue_s(j + 1, last);
            }
            ok = ok && mbar_wait(&v_full[vs.s], vs.ph, abort_flag) && mbar_wait(&p_full[x], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < kBM / 16; ++kk)
              umma_ts_h(o_col, p_col + kk * 8, dv_, vs.s * C::TILE_BYTES + kk * (16 * 128), idesc, (j > 0 || kk > 0) ? 1u : 0u);
            umma_commit(&pv_done[x]);
            umma_commit(&v_empty[vs.s]);
            vs.next();
            if (!C::P_APART && j < last) issue_s(j + 1, last);  // over the P just read: the tensor core keeps the order
            ph ^= 1u;
          }
          for (int j = last + 1; j < q1 && ok; ++j) skip();
          work.next();
          last = work.valid ? last_of(work) : -1;
          if (last >= 0) issue_s(0, last);  // S has been read: P of it has been multiplied
        }
        if (!ok) {
          *abort_flag = 1;
          if (p.status) atomicCAS(p.status, 0, kStatusMmaTimeout);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, stores
    // Quadrant = warp & 3 (query rows), x = which query tile.  A wait that gives up raises the abort flag for all roles
    // and the warp goes on (its lanes stay together); nothing is stored then.
    take_registers<96, 200>();
    const int quad = warp & 3;
    const int x = (warp - 4) >> 2;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t s_col = lane_base + C::S_COL + x * kBM, p_col = lane_base + C::P_COL + x * C::P_TILE;
    const uint32_t o_col = C::O_COL + x * D;
    const f32x2 s2 = pack2(p.scale_log2, p.scale_log2);
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (!mbar_wait(bar, parity, abort_flag)) *abort_flag = 1;
      __syncwarp();  // the tensor-memory accesses that follow take the whole warp at once
    };
    uint32_t ph = 0;  // of the tile at hand: s_full, s_free, p_full, pv_done
    for (; work.valid;) {
      const int qt = (items - 1 - work.level) * p.pair + x;
      const int b = p.by_heads(work.head), h = work.head - b * p.H;
      work.next();
      if (x >= p.pair || qt >= tiles) continue;
      float m_used = -INFINITY;  // reference max of the exponentials accumulated so far (log2 domain)
      float l = 0.f;
      for (int j = 0; j <= qt; ++j) {
        wait(&s_full[x], ph);
        tc_fence_after();
        float sc[kBM];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_col + c * 32, *reinterpret_cast<float(*)[32]>(&sc[c * 32]));
        tmem_ld_wait();
        if (C::P_APART) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_free[x]);
        }
        if (j == qt) {
#pragma unroll
          for (int i = 0; i < kBM; ++i)
            if (i > row_in_tile) sc[i] = -INFINITY;
        }
        // row maximum of the raw scores (the scale is positive), four independent chains
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < kBM; i += 8) {
#pragma unroll
          for (int t = 0; t < 4; ++t) mx4[t] = fmaxf(mx4[t], fmaxf(sc[i + 2 * t], sc[i + 2 * t + 1]));
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
        const float m_new = fmaxf(m_used, mx);
        const bool need = (j == 0) || (m_new - m_used > kRescaleThreshold);
        if (__any_sync(0xffffffffu, need)) {
          if (j > 0) {
            // O may only be touched between two products: the one before must have retired, the next one cannot start
            // before this warp delivered its P
            wait(&pv_done[x], ph ^ 1u);
            tc_fence_after();
            const float alpha = (m_new == -INFINITY) ? 1.f : fast_exp2(m_used - m_new);
            l *= alpha;
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              float o[32];
              tmem_ld_32x32(lane_base + o_col + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] *= alpha;
              tmem_st_32x32(lane_base + o_col + c * 32, o);
            }
            tmem_st_wait();
          }
          m_used = m_new;
        }
        const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
        const f32x2 nm2 = pack2(neg_m, neg_m);
        f32x2 sums[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
        // exponentials, packed to bf16 pairs
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float e0, e1;
            unpack2(fma2(pack2(sc[c * 32 + i], sc[c * 32 + i + 1]), s2, nm2), e0, e1);
            e0 = fast_exp2(e0);
            e1 = fast_exp2(e1);
            pk[i >> 1] = pack_bf16x2(e0, e1);
            sums[(i >> 1) & 1] = add2(sums[(i >> 1) & 1], pack2(e0, e1));
          }
          if (C::P_APART && c == 0) wait(&pv_done[x], ph ^ 1u);  // the P before this one
          tmem_st_32x16(p_col + c * 16, pk);
        }
        float sum0, sum1;
        unpack2(add2(sums[0], sums[1]), sum0, sum1);
        l += sum0 + sum1;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[x]);
        ph ^= 1u;
      }
      // normalise, write out and the log-sum-exp.  The next item's first product overwrites O only after these warps
      // delivered its P.
      wait(&pv_done[x], ph ^ 1u);
      tc_fence_after();
      if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
      const int rows = p.T - qt * kBM;
      store_rows<D, true>(tmem_base + o_col, quad, lane, p.out + (((long long)b * p.T + qt * kBM) * p.H + h) * D,
                          (long long)p.H * D, rows, l > 0.f ? 1.f / l : 0.f);
      if (row_in_tile < rows)
        p.lse[((long long)b * p.H + h) * p.T + qt * kBM + row_in_tile] =
            (l > 0.f) ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
    if (*abort_flag != 0 && lane == 0 && p.status) atomicCAS(p.status, 0, kStatusEpilogueTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    // a wait gave up: let copies that are still in flight land before the CTA retires
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// ============================================================================================ backward
// dQ, dK, dV of causal attention from q, k, v, dO, the forward's log-sum-exp and delta_i = sum_d O_id dO_id.  With
// S = scale * Q K^T, P = exp(S - lse):
//   dV = P^T dO,  dP = dO V^T,  dS = P o (dP - delta) * scale,  dQ = dS K,  dK = dS^T Q.
// Two kernels, neither needs atomics: attn_bwd_dq_kernel loops over the kv tiles of a query tile, attn_bwd_dkv_kernel over
// the query tiles of a kv tile and over the query heads that share the kv head.  P and dS are rebuilt in registers from S
// and dP and handed to the next MMA as bf16 through tensor memory.

struct AttnBwdParams {
  __nv_bfloat16* dq;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  const float* neg_lse2;   // see attn_delta_kernel
  const float* neg_delta;
  int B, T, H, Hkv;
  WorkPlan q_plan, kv_plan;
  FastDiv by_heads, by_kv_heads, by_group;
  float scale, scale_log2;
  int* status;
};

// What the backward kernels take per query row, laid out [B, H, T rounded up to 128]:
//   neg_lse2 = -lse * log2(e) (-inf beyond the sequence: P is zero there),  neg_delta = -scale * sum_d O_d dO_d.
// D / 8 lanes per row, 16 bytes per lane, two rows per lane; a block takes consecutive rows of one head, so that what it
// writes is contiguous (64 x 1024 rows of 12 heads of 64: 45 us with the rows of a block spread over the heads).
constexpr int kDeltaRows = 2;  // per lane
template <int D>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o,
                                                        const __nv_bfloat16* __restrict__ d_o,
                                                        const float* __restrict__ lse, float* __restrict__ neg_lse2,
                                                        float* __restrict__ neg_delta, int T, int H, int t_pad,
                                                        FastDiv by_heads, float scale) {
  pdl_trigger();
  pdl_wait();
  constexpr int LPR = D / 8;  // lanes per row: 16 (D = 128) or 8 (D = 64)
  constexpr int ROWS = 256 / LPR;
  const int sub = threadIdx.x % LPR;
  const int bh = (int)blockIdx.x, b = by_heads(bh), h = bh - b * H;
  const int t0 = (int)blockIdx.y * (ROWS * kDeltaRows) + threadIdx.x / LPR;
  uint4 a[kDeltaRows], g[kDeltaRows];
#pragma unroll
  for (int r = 0; r < kDeltaRows; ++r) {
    const int t = t0 + r * ROWS;
    const long long src = (((long long)b * T + t) * H + h) * D + sub * 8;
    a[r] = t < T ? *reinterpret_cast<const uint4*>(o + src) : make_uint4(0, 0, 0, 0);
    g[r] = t < T ? *reinterpret_cast<const uint4*>(d_o + src) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int r = 0; r < kDeltaRows; ++r) {
    const int t = t0 + r * ROWS;
    const __nv_bfloat162* ah = reinterpret_cast<const __nv_bfloat162*>(&a[r]);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g[r]);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(ah[i]), y = __bfloat1622float2(gh[i]);
      s = fmaf(x.x, y.x, fmaf(x.y, y.y, s));
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (sub == 0 && t < t_pad) {
      const long long dst = (long long)bh * t_pad + t;
      neg_delta[dst] = t < T ? -s * scale : 0.f;
      neg_lse2[dst] = t < T ? -lse[(long long)bh * T + t] * 1.4426950408889634f : -INFINITY;
    }
  }
}

// ---------------------------------------------------------------------------------- dQ
constexpr int kDqThreads = 32 * 12;  // TMA; S, dP and dQ; two spare; eight softmax warps (two per lane quadrant, 64 columns each)

template <int D>
struct BwdQCfg {
  static constexpr int PANELS = D / 64;
  static constexpr int TILE_BYTES = kBM * D * 2;  // 128 rows of Q, dO, K or V
  static constexpr int K_STAGES = D == 128 ? 3 : 4, V_STAGES = D == 128 ? 2 : 4;
  static constexpr int SMEM = (2 + K_STAGES + V_STAGES) * TILE_BYTES + 256;
  // tensor memory: S, dP, two buffers of dS, dQ; D = 64 has room for Q and dO too (as A operands they leave half of the
  // shared memory's bandwidth to the rest)
  static constexpr bool Q_IN_TMEM = D == 64;
  static constexpr int S_COL = 0, DP_COL = kBM, DS_COL = 2 * kBM, DQ_COL = 3 * kBM;
  static constexpr int Q_COL = DQ_COL + D, DO_COL = Q_COL + D / 2;
  static constexpr int TMEM_COLS = 512;
  static_assert((Q_IN_TMEM ? DO_COL + D / 2 : DQ_COL + D) <= TMEM_COLS && SMEM <= 232448, "one CTA per SM");
};

// One CTA per SM runs through (query tile of 128 rows) x (kv tiles of 128 rows that it sees).  The softmax warps load S
// and dP of a tile into registers at once and release both, so the next tile's products run under the 1024 cycles that the
// exponentials of this one take; dS alternates between two buffers, and the products of tile i + 1 are issued after
// dQ += dS K of tile i - 1, so whoever sees S of tile i + 1 may overwrite the dS of tile i - 1.
template <int D>
__global__ void __launch_bounds__(kDqThreads, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_do,
                   const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                   const AttnBwdParams p) {
  using C = BwdQCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sDO = sQ + C::TILE_BYTES;
  uint8_t* sK = sDO + C::TILE_BYTES;
  uint8_t* sV = sK + C::K_STAGES * C::TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + C::V_STAGES * C::TILE_BYTES);
  uint64_t* q_full = bars;       // Q and dO
  uint64_t* q_empty = bars + 1;
  uint64_t* sdp_full = bars + 2;
  uint64_t* sdp_free = bars + 3;  // softmax warps: S and dP are in registers
  uint64_t* ds_full = bars + 4;   // softmax warps; one per buffer of dS: a warp may deliver the next tile's before another
                                  // has delivered this one's, as S and dP are released before dS is formed
  uint64_t* dq_full = bars + 6;
  uint64_t* k_full = bars + 7;    // K_STAGES each
  uint64_t* k_empty = k_full + C::K_STAGES;
  uint64_t* v_full = k_empty + C::K_STAGES;  // V_STAGES each
  uint64_t* v_empty = v_full + C::V_STAGES;
  uint64_t* bars_end = v_empty + C::V_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_end);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = (int)warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int tiles = (p.T + kBM - 1) / kBM;
  WorkList work(p.q_plan);          // level 0 = the last query tile, which sees all kv tiles
  if (smem_u32(smem) & 1023) {      // the 128-byte swizzle repeats every 1024 bytes
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, kStatusBadArgument);
    return;
  }

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_do);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    for (uint64_t* b = bars; b < bars_end; ++b) mbar_init(b, (b >= sdp_free && b < dq_full) ? 8 : 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  pdl_trigger();
  pdl_wait();
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  if (warp < 4) {
    give_registers<72, 216>();
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      if (lane == 0) {
        bool ok = true;
        Ring<C::K_STAGES> ks;
        Ring<C::V_STAGES> vs;
        auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col, int row, int seq) {
#pragma unroll
          for (int c = 0; c < C::PANELS; ++c) tma_load_3d(dst + c * (kBM * 128), map, bar, col + c * 64, row, seq);
        };
        for (int r = 0; ok && work.valid; ++r, work.next()) {
          const int qt = tiles - 1 - work.level, b = p.by_heads(work.head), h = work.head - b * p.H, hk = p.by_group(h);
          ok = mbar_wait(q_empty, (r & 1) ^ 1u, abort_flag);
          if (!ok) break;
          mbar_arrive_expect_tx(q_full, 2 * C::TILE_BYTES);
          load(sQ, &tmap_q, q_full, h * D, qt * kBM, b);
          load(sDO, &tmap_do, q_full, h * D, qt * kBM, b);
          for (int j = 0; j <= qt; ++j) {
            ok = mbar_wait(&k_empty[ks.s], ks.ph ^ 1u, abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(&k_full[ks.s], C::TILE_BYTES);
            load(sK + ks.s * C::TILE_BYTES, &tmap_k, &k_full[ks.s], hk * D, j * kBM, b);
            ok = mbar_wait(&v_empty[vs.s], vs.ph ^ 1u, abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(&v_full[vs.s], C::TILE_BYTES);
            load(sV + vs.s * C::TILE_BYTES, &tmap_v, &v_full[vs.s], hk * D, j * kBM, b);
            ks.next();
            vs.next();
          }
        }
        if (!ok) {
          *abort_flag = 1;
          if (p.status) atomicCAS(p.status, 0, kStatusProducerTimeout);
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- S = Q K^T, dP = dO V^T, dQ += dS K
      if (elect_one()) {
        constexpr uint32_t idesc_dq = make_instr_desc(1, kMajorK, kMajorMN, kBM, D);
        const DescHalves dq_ = desc_halves(smem_u32(sQ), 16, 1024), ddo_ = desc_halves(smem_u32(sDO), 16, 1024);
        const DescHalves dk_ = desc_halves(smem_u32(sK), 16, 1024), dv_ = desc_halves(smem_u32(sV), 16, 1024);
        const DescHalves dkm_ = desc_halves(smem_u32(sK), kBM * 128, 1024);  // K as [kv rows (K)] x [D (N)], MN-major
        bool ok = true;
        Ring<C::K_STAGES> ks, ka;  // S; dQ
        Ring<C::V_STAGES> vs;
        uint32_t ph = 0, n_a = 0;  // parity of the next S; dQ products so far
        // dQ of the tile before: its dS lies in buffer n_a & 1
        auto accumulate = [&](bool fresh, bool last) -> bool {
          if (!mbar_wait(&ds_full[n_a & 1], (n_a >> 1) & 1, abort_flag)) return false;
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < kBM / 16; ++kk)
            umma_ts_h(tmem_base + C::DQ_COL, tmem_base + C::DS_COL + (n_a & 1) * 64 + kk * 8, dkm_,
                      ka.s * C::TILE_BYTES + kk * (16 * 128), idesc_dq, (!fresh || kk > 0) ? 1u : 0u);
          umma_commit(&k_empty[ka.s]);
          if (last) umma_commit(dq_full);
          ka.next();
          ++n_a;
          return true;
        };
        int behind = 0;  // kv tiles of the query tile before whose dQ is outstanding: its last one
        bool behind_fresh = false;
        for (int r = 0; ok && work.valid; ++r, work.next()) {
          const int n = tiles - work.level;
          for (int j = 0; j < n; ++j) {
            ok = (j > 0 || mbar_wait(q_full, r & 1, abort_flag)) && mbar_wait(&k_full[ks.s], ks.ph, abort_flag) &&
                 mbar_wait(&v_full[vs.s], vs.ph, abort_flag) && mbar_wait(sdp_free, ph ^ 1u, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (C::Q_IN_TMEM && j == 0) {  // the S and dP before these have been read
              keep_tile<D>(tmem_base + C::Q_COL, dq_);
              keep_tile<D>(tmem_base + C::DO_COL, ddo_);
              umma_commit(q_empty);
            }
            scores<D, C::Q_IN_TMEM>(tmem_base + C::S_COL, dq_, tmem_base + C::Q_COL, dk_, ks.s * C::TILE_BYTES);
            scores<D, C::Q_IN_TMEM>(tmem_base + C::DP_COL, ddo_, tmem_base + C::DO_COL, dv_, vs.s * C::TILE_BYTES);
            umma_commit(sdp_full);
            umma_commit(&v_empty[vs.s]);
            if (!C::Q_IN_TMEM && j == n - 1) umma_commit(q_empty);
            ks.next();
            vs.next();
            ph ^= 1u;
            if (behind) {
              ok = accumulate(behind_fresh, j == 0);
              if (!ok) break;
            }
            behind = 1;
            behind_fresh = j == 0;
          }
        }
        if (ok && behind) ok = accumulate(behind_fresh, true);
        if (!ok) {
          *abort_flag = 1;
          if (p.status) atomicCAS(p.status, 0, kStatusMmaTimeout);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, stores
    // Quadrant = warp & 3 (query rows), half = which 64 of the 128 kv columns.  A wait that gives up raises the abort flag
    // for all roles and the warp goes on (its lanes stay together); nothing is stored then.
    take_registers<72, 216>();
    const int quad = warp & 3;
    const int half = (warp - 4) >> 2;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
    const f32x2 scale2 = pack2(p.scale_log2, p.scale_log2), out_scale2 = pack2(p.scale, p.scale);
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (!mbar_wait(bar, parity, abort_flag)) *abort_flag = 1;
      __syncwarp();  // the tensor-memory accesses that follow take the whole warp at once
    };
    uint32_t ph = 0;
    for (int r = 0; work.valid; ++r) {
      const int qt = tiles - 1 - work.level, b = p.by_heads(work.head), h = work.head - b * p.H;
      const long long stat = (long long)work.head * tiles * kBM + qt * kBM + row_in_tile;
      const float nl = p.neg_lse2[stat], nd = p.neg_delta[stat];
      const f32x2 nl2 = pack2(nl, nl), nd2 = pack2(nd, nd);
      for (int j = 0; j <= qt; ++j) {
        wait(sdp_full, ph);
        tc_fence_after();
        float sc[64], dp[64];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          tmem_ld_32x32(lane_base + C::S_COL + half * 64 + q * 32, *reinterpret_cast<float(*)[32]>(&sc[q * 32]));
          tmem_ld_32x32(lane_base + C::DP_COL + half * 64 + q * 32, *reinterpret_cast<float(*)[32]>(&dp[q * 32]));
        }
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(sdp_free);
        // dS = P o (dP - delta) * scale
        float pk[32];
        auto columns = [&](auto masked) {
#pragma unroll
          for (int c = 0; c < 64; c += 2) {
            float p0, p1, d0, d1;
            unpack2(fma2(pack2(sc[c], sc[c + 1]), scale2, nl2), p0, p1);
            p0 = fast_exp2(p0);
            p1 = fast_exp2(p1);
            if constexpr (decltype(masked)::value) {
              if (half * 64 + c > row_in_tile) p0 = 0.f;
              if (half * 64 + c + 1 > row_in_tile) p1 = 0.f;
            }
            unpack2(mul2(pack2(p0, p1), fma2(pack2(dp[c], dp[c + 1]), out_scale2, nd2)), d0, d1);
            pk[c >> 1] = __uint_as_float(pack_bf16x2(d0, d1));
          }
        };
        if (j == qt) columns(std::true_type());
        else columns(std::false_type());
        tmem_st_32x32(lane_base + C::DS_COL + ph * 64 + half * 32, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_full[ph]);
        ph ^= 1u;
      }
      work.next();
      wait(dq_full, r & 1);
      tc_fence_after();
      if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
      // half of the columns each; the next query tile's first product overwrites dQ only after these warps delivered its dS
      store_rows<D / 2>(tmem_base + C::DQ_COL + half * (D / 2), quad, lane,
                        p.dq + (((long long)b * p.T + qt * kBM) * p.H + h) * D + half * (D / 2), (long long)p.H * D,
                        p.T - qt * kBM);
    }
    if (*abort_flag != 0 && lane == 0 && p.status) atomicCAS(p.status, 0, kStatusEpilogueTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    // a wait gave up: let copies that are still in flight land before the CTA retires
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------- dK, dV
constexpr int kSoftmaxWarps = 16;                  // four per lane quadrant, each with 32 of a tile's 128 columns
constexpr int kBwdThreads = 32 * (4 + kSoftmaxWarps);  // TMA; S^T; dV, dK; dP^T; softmax

template <int D>
struct BwdKvCfg {
  static constexpr int PANELS = D / 64;
  static constexpr int TILE_BYTES = kBM * D * 2;    // 128 rows of K, V, Q or dO
  static constexpr int STAT_BYTES = kBM * 4;        // one fp32 per query row
  static constexpr int Q_STAGES = D == 128 ? 3 : 4;   // query-side tiles in flight
  static constexpr int DO_STAGES = D == 128 ? 2 : 4;
  static constexpr int SMEM = (2 + Q_STAGES + DO_STAGES) * TILE_BYTES + (Q_STAGES + DO_STAGES) * STAT_BYTES + 256;
  // Tensor memory.  D = 64 keeps K and V there too (as A operands they leave half of the shared memory's bandwidth to
  // the rest) and P^T beside S^T; at D = 128 dV and dK take half of it, P^T is written over S^T.
  static constexpr bool KV_IN_TMEM = D == 64;
  static constexpr int S_COL = 0, DP_COL = kBM;
  static constexpr int P_COL = KV_IN_TMEM ? 2 * kBM : S_COL;
  static constexpr int P_STEP = KV_IN_TMEM ? 16 : 32;  // columns from the P^T of 32 query rows to that of the next 32
  static constexpr int DV_COL = KV_IN_TMEM ? 2 * kBM + 64 : 2 * kBM;
  static constexpr int DK_COL = DV_COL + D;
  static constexpr int K_COL = DK_COL + D, V_COL = K_COL + D / 2;
  static constexpr int TMEM_COLS = 512;
  static_assert((KV_IN_TMEM ? V_COL + D / 2 : DK_COL + D) <= TMEM_COLS && SMEM <= 232448, "one CTA per SM");
};

// One CTA per SM runs through (kv tile of 128 rows) x (query tiles of 128 rows that see it, over the query heads of the
// kv head).  Per pair of tiles the tensor core multiplies for 1024 cycles (D = 64; 2048 at D = 128) and the special
// function unit takes 1024 for the exponentials; the order below keeps both fed: while the softmax warps turn S^T of one
// tile into P^T, the tensor core runs dK and dP^T of the tile before, and dV and the next S^T while they form dS^T.
// P^T and dS^T go back over the columns that the same thread read (D = 64 has room for P^T beside S^T), so no warp waits for
// another.  The next kv tile's loads and first products run under the last tile of the one before; only the store of dV and dK
// stands alone.
template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_do,
                    const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                    const AttnBwdParams p) {
  using C = BwdKvCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = sK + C::TILE_BYTES;
  uint8_t* sQ = sV + C::TILE_BYTES;
  uint8_t* sDO = sQ + C::Q_STAGES * C::TILE_BYTES;
  float* sLse = reinterpret_cast<float*>(sDO + C::DO_STAGES * C::TILE_BYTES);  // -lse * log2(e) of each stage's rows
  float* sDelta = sLse + C::Q_STAGES * kBM;                                    // -delta * scale
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDelta + C::DO_STAGES * kBM);
  uint64_t* k_full = bars;       // 1
  uint64_t* k_empty = bars + 1;  // 1
  uint64_t* v_full = bars + 2;   // 1
  uint64_t* v_empty = bars + 3;  // 1
  uint64_t* s_full = bars + 4;
  uint64_t* s_free = bars + 5;   // softmax warps: S^T is in registers (KV_IN_TMEM)
  uint64_t* p_full = bars + 6;   // softmax warps
  uint64_t* dp_full = bars + 7;
  uint64_t* ds_full = bars + 8;  // softmax warps
  uint64_t* dv_done = bars + 9;  // P^T has been multiplied
  uint64_t* dk_done = bars + 10;  // dS^T has been multiplied
  uint64_t* acc_full = bars + 11;
  uint64_t* q_full = bars + 12;   // Q_STAGES each
  uint64_t* q_empty = q_full + C::Q_STAGES;
  uint64_t* do_full = q_empty + C::Q_STAGES;  // DO_STAGES each
  uint64_t* do_empty = do_full + C::DO_STAGES;  // both MMA warps
  uint64_t* bars_end = do_empty + C::DO_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars_end);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = (int)warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int tiles = (p.T + kBM - 1) / kBM;
  const int group = p.H / p.Hkv;
  WorkList work(p.kv_plan);  // level = kv tile: the first one is seen by all query tiles
  if (smem_u32(smem) & 1023) {  // the 128-byte swizzle repeats every 1024 bytes
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, kStatusBadArgument);
    return;
  }

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_do);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    for (uint64_t* b = bars; b < bars_end; ++b)
      mbar_init(b, (b == ds_full || b == p_full || b == s_free) ? kSoftmaxWarps : b >= do_empty ? 2 : 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  pdl_trigger();
  pdl_wait();
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      bool ok = true;
      Ring<C::Q_STAGES> qs;
      Ring<C::DO_STAGES> os;
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col, int row, int seq) {
#pragma unroll
        for (int c = 0; c < C::PANELS; ++c) tma_load_3d(dst + c * (kBM * 128), map, bar, col + c * 64, row, seq);
      };
      for (int r = 0; ok && work.valid; ++r, work.next()) {
        const int kt = work.level, b = p.by_kv_heads(work.head), hk = work.head - b * p.Hkv;
        ok = mbar_wait(k_empty, (r & 1) ^ 1u, abort_flag);
        if (!ok) break;
        mbar_arrive_expect_tx(k_full, C::TILE_BYTES);
        load(sK, &tmap_k, k_full, hk * D, kt * kBM, b);
        for (int g = 0; g < group && ok; ++g) {
          const int h = hk * group + g;
          const long long stat0 = ((long long)b * p.H + h) * ((long long)tiles * kBM);
          for (int i = kt; i < tiles && ok; ++i) {
            ok = mbar_wait(&q_empty[qs.s], qs.ph ^ 1u, abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(&q_full[qs.s], C::TILE_BYTES + C::STAT_BYTES);
            load(sQ + qs.s * C::TILE_BYTES, &tmap_q, &q_full[qs.s], h * D, i * kBM, b);
            bulk_load_1d(sLse + qs.s * kBM, p.neg_lse2 + stat0 + i * kBM, C::STAT_BYTES, &q_full[qs.s]);
            if (g == 0 && i == kt) {
              ok = mbar_wait(v_empty, (r & 1) ^ 1u, abort_flag);
              if (!ok) break;
              mbar_arrive_expect_tx(v_full, C::TILE_BYTES);
              load(sV, &tmap_v, v_full, hk * D, kt * kBM, b);
            }
            ok = mbar_wait(&do_empty[os.s], os.ph ^ 1u, abort_flag);
            if (!ok) break;
            mbar_arrive_expect_tx(&do_full[os.s], C::TILE_BYTES + C::STAT_BYTES);
            load(sDO + os.s * C::TILE_BYTES, &tmap_do, &do_full[os.s], h * D, i * kBM, b);
            bulk_load_1d(sDelta + os.s * kBM, p.neg_delta + stat0 + i * kBM, C::STAT_BYTES, &do_full[os.s]);
            qs.next();
            os.next();
          }
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.status) atomicCAS(p.status, 0, kStatusProducerTimeout);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ S^T = K Q^T
    if (elect_one()) {
      const DescHalves dk_ = desc_halves(smem_u32(sK), 16, 1024), dq_ = desc_halves(smem_u32(sQ), 16, 1024);
      bool ok = true;
      Ring<C::Q_STAGES> qs;
      uint32_t ph = 0;
      for (int r = 0; ok && work.valid; ++r, work.next()) {
        const int n = (tiles - work.level) * group;
        for (int i = 0; i < n; ++i) {
          ok = (i > 0 || mbar_wait(k_full, r & 1, abort_flag)) && mbar_wait(&q_full[qs.s], qs.ph, abort_flag) &&
               mbar_wait(C::KV_IN_TMEM ? s_free : dv_done, ph ^ 1u, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (C::KV_IN_TMEM && i == 0) {
            keep_tile<D>(tmem_base + C::K_COL, dk_);  // the S^T before this one has been read
            umma_commit(k_empty);
          }
          scores<D, C::KV_IN_TMEM>(tmem_base + C::S_COL, dk_, tmem_base + C::K_COL, dq_, qs.s * C::TILE_BYTES);
          umma_commit(s_full);
          if (!C::KV_IN_TMEM && i == n - 1) umma_commit(k_empty);
          ph ^= 1u;
          qs.next();
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.status) atomicCAS(p.status, 0, kStatusMmaTimeout);
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ dP^T = V dO^T
    if (elect_one()) {
      const DescHalves dv_ = desc_halves(smem_u32(sV), 16, 1024), ddo_ = desc_halves(smem_u32(sDO), 16, 1024);
      bool ok = true;
      Ring<C::DO_STAGES> os;
      uint32_t ph = 0;
      for (int r = 0; ok && work.valid; ++r, work.next()) {
        const int n = (tiles - work.level) * group;
        for (int i = 0; i < n; ++i) {
          ok = (i > 0 || mbar_wait(v_full, r & 1, abort_flag)) && mbar_wait(&do_full[os.s], os.ph, abort_flag) &&
               mbar_wait(dk_done, ph ^ 1u, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (C::KV_IN_TMEM && i == 0) {
            keep_tile<D>(tmem_base + C::V_COL, dv_);
            umma_commit(v_empty);
          }
          scores<D, C::KV_IN_TMEM>(tmem_base + C::DP_COL, dv_, tmem_base + C::V_COL, ddo_, os.s * C::TILE_BYTES);
          umma_commit(dp_full);
          umma_commit(&do_empty[os.s]);
          if (!C::KV_IN_TMEM && i == n - 1) umma_commit(v_empty);
          ph ^= 1u;
          os.next();
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.status) atomicCAS(p.status, 0, kStatusMmaTimeout);
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ accumulators: dV += P^T dO, dK += dS^T Q
    if (elect_one()) {
      constexpr uint32_t idesc = make_instr_desc(1, kMajorK, kMajorMN, kBM, D);
      const DescHalves dq_ = desc_halves(smem_u32(sQ), kBM * 128, 1024), ddo_ = desc_halves(smem_u32(sDO), kBM * 128, 1024);
      // A: bf16 pairs in tensor memory, 32 query rows every a_step columns
      auto accumulate = [&](uint32_t col, uint32_t a_col, uint32_t a_step, DescHalves b, uint32_t b_off, bool fresh) {
#pragma unroll
        for (int kk = 0; kk < kBM / 16; ++kk)
          umma_ts_h(tmem_base + col, tmem_base + a_col + (kk >> 1) * a_step + (kk & 1) * 8, b, b_off + kk * (16 * 128), idesc,
                    (!fresh || kk > 0) ? 1u : 0u);
      };
      bool ok = true;
      Ring<C::Q_STAGES> qs;
      Ring<C::DO_STAGES> os;
      uint32_t ph = 0;
      for (; ok && work.valid; work.next()) {
        const int n = (tiles - work.level) * group;
        for (int i = 0; i < n; ++i) {
          ok = mbar_wait(&do_full[os.s], os.ph, abort_flag) && mbar_wait(p_full, ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          accumulate(C::DV_COL, C::P_COL, C::P_STEP, ddo_, os.s * C::TILE_BYTES, i == 0);
          umma_commit(dv_done);
          ok = mbar_wait(ds_full, ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          accumulate(C::DK_COL, C::DP_COL, 32, dq_, qs.s * C::TILE_BYTES, i == 0);
          umma_commit(dk_done);
          umma_commit(&q_empty[qs.s]);
          umma_commit(&do_empty[os.s]);  // not before: the softmax read delta_i from this stage up to its dS^T
          if (i == n - 1) umma_commit(acc_full);
          ph ^= 1u;
          qs.next();
          os.next();
        }
      }
      if (!ok) {
        *abort_flag = 1;
        if (p.status) atomicCAS(p.status, 0, kStatusMmaTimeout);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax, stores
    // Quadrant = warp & 3 (kv rows), part = which 32 of the 128 query columns.  A wait that gives up raises the abort flag
    // for all roles and the warp goes on (its lanes stay together); nothing is stored then.
    const int quad = warp & 3;
    const int part = (warp - 4) >> 2;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
    const f32x2 scale2 = pack2(p.scale_log2, p.scale_log2), out_scale2 = pack2(p.scale, p.scale);
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (!mbar_wait(bar, parity, abort_flag)) *abort_flag = 1;
      __syncwarp();  // the tensor-memory accesses that follow take the whole warp at once
    };
    Ring<C::Q_STAGES> qs;
    Ring<C::DO_STAGES> os;
    uint32_t ph = 0;
    for (int r = 0; work.valid; ++r) {
      const int kt = work.level, b = p.by_kv_heads(work.head), hk = work.head - b * p.Hkv;
      for (int g = 0; g < group; ++g) {
        for (int i = kt; i < tiles; ++i) {
          // P = exp(S * scale - lse), kept in registers for dS
          wait(s_full, ph);
          tc_fence_after();
          float pr[32];
          tmem_ld_32x32(lane_base + C::S_COL + part * 32, pr);
          tmem_ld_wait();
          if (C::KV_IN_TMEM) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_free);
          }
          const float* lse_s = sLse + qs.s * kBM + part * 32;
          {
            uint32_t pk[16];
            auto columns = [&](auto masked) {
#pragma unroll
              for (int c = 0; c < 32; c += 4) {
                const float4 l4 = *reinterpret_cast<const float4*>(lse_s + c);
#pragma unroll
                for (int t = 0; t < 4; t += 2) {
                  float e0, e1;
                  unpack2(fma2(pack2(pr[c + t], pr[c + t + 1]), scale2, t ? pack2(l4.z, l4.w) : pack2(l4.x, l4.y)), e0, e1);
                  e0 = fast_exp2(e0);
                  e1 = fast_exp2(e1);
                  if constexpr (decltype(masked)::value) {
                    if (part * 32 + c + t < row_in_tile) e0 = 0.f;
                    if (part * 32 + c + t + 1 < row_in_tile) e1 = 0.f;
                  }
                  pr[c + t] = e0;
                  pr[c + t + 1] = e1;
                  pk[(c + t) >> 1] = pack_bf16x2(e0, e1);
                }
              }
            };
            if (i == kt) columns(std::true_type());
            else columns(std::false_type());
            if (C::KV_IN_TMEM) wait(dv_done, ph ^ 1u);  // the P^T before this one
            tmem_st_32x16(lane_base + C::P_COL + part * C::P_STEP, pk);
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full);
          // dS = P o (dP - delta) * scale
          wait(dp_full, ph);
          tc_fence_after();
          {
            const float* dlt_s = sDelta + os.s * kBM + part * 32;
            float dp[32];
            uint32_t dk[16];
            tmem_ld_32x32(lane_base + C::DP_COL + part * 32, dp);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
              const float4 d4 = *reinterpret_cast<const float4*>(dlt_s + c);
#pragma unroll
              for (int t = 0; t < 4; t += 2) {
                const f32x2 d = fma2(pack2(dp[c + t], dp[c + t + 1]), out_scale2, t ? pack2(d4.z, d4.w) : pack2(d4.x, d4.y));
                float g0, g1;
                unpack2(mul2(pack2(pr[c + t], pr[c + t + 1]), d), g0, g1);
                dk[(c + t) >> 1] = pack_bf16x2(g0, g1);
              }
            }
            tmem_st_32x16(lane_base + C::DP_COL + part * 32, dk);
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(ds_full);
          ph ^= 1u;
          qs.next();
          os.next();
        }
      }
      work.next();
      wait(acc_full, r & 1);
      tc_fence_after();
      if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
      // Parts 0 and 1 write dV, 2 and 3 dK, half of the columns each.  The next kv tile's products overwrite both only
      // after these warps delivered its first P^T and dS^T, which they do after the reads here.
      const int c0 = (part & 1) * (D / 2);
      __nv_bfloat16* base = (part < 2 ? p.dv : p.dk) + (((long long)b * p.T + kt * kBM) * p.Hkv + hk) * D + c0;
      store_rows<D / 2>(tmem_base + (part < 2 ? C::DV_COL : C::DK_COL) + c0, quad, lane, base, (long long)p.Hkv * D,
                        p.T - kt * kBM);
    }
    if (*abort_flag != 0 && lane == 0 && p.status) atomicCAS(p.status, 0, kStatusEpilogueTimeout);
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn attn_encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(sym);
  });
  return fn;
}

// [seqs, T, cols] bf16, contiguous; box = 64 columns x kBM rows of one sequence (rows beyond T read as zeros), 128-byte swizzle
bool attn_tmap_seq(CUtensorMap* map, const void* base, uint64_t cols, uint64_t T, uint64_t seqs) {
  EncodeFn fn = attn_encode_fn();
  if (!fn || (reinterpret_cast<uintptr_t>(base) & 15)) return false;
  cuuint64_t dims[3] = {cols, T, seqs};
  cuuint64_t strides[2] = {cols * 2, T * cols * 2};
  cuuint32_t box[3] = {64, kBM, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  auto encode = [&] {
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT && bind_primary_context()) r = encode();  // the first call of a thread
  return r == CUDA_SUCCESS;
}

// CTAs of a persistent kernel with one CTA per SM
int attn_grid(long long items) {
  static std::atomic<int> known[64];  // per device; the count does not change
  int dev = 0;
  cudaGetDevice(&dev);
  int sms = dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
  if (sms == 0) {
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    if (dev < 64) known[dev].store(sms, std::memory_order_relaxed);
  }
  return (int)(items < sms ? items : sms);
}

template <int D>
cudaError_t attn_fwd_launch_d(const void* q, const void* k, const void* v, void* out, float* lse, int B, int T, int H,
                              int Hkv, float scale, int* status, cudaStream_t stream) {
  using C = AttnCfg<D>;
  CUtensorMap tq, tk, tv;
  if (!attn_tmap_seq(&tq, q, (uint64_t)H * D, T, B) || !attn_tmap_seq(&tk, k, (uint64_t)Hkv * D, T, B) ||
      !attn_tmap_seq(&tv, v, (uint64_t)Hkv * D, T, B))
    return cudaErrorInvalidValue;
  auto kernel = attn_fwd_kernel<D>;
  static std::atomic<unsigned long long> granted{0};
  const cudaError_t e = once_per_device(granted, [&] {
    cudaFuncAttributes fa;
    // the register shares of the kernel's warps add up to what it is launched with, or the larger one waits forever
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess || fa.numRegs != 168) return cudaErrorInvalidConfiguration;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  });
  if (e != cudaSuccess) return e;
  AttnParams p;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.B = B;
  p.T = T;
  p.H = H;
  p.Hkv = Hkv;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  const int tiles = (T + kBM - 1) / kBM;
  const int heads = B * H, sms = attn_grid(1 << 20);
  p.pair = (long long)heads * tiles > sms ? 2 : 1;
  const int items = (tiles + p.pair - 1) / p.pair, ctas = attn_grid((long long)heads * items);
  p.plan = WorkPlan(items, heads, ctas);
  p.by_heads = FastDiv(H);
  p.by_group = FastDiv(H / Hkv);
  launch_pdl(kernel, dim3(ctas), dim3(kFwdThreads), C::SMEM, stream, 0, tq, tk, tv, p);
  return cudaGetLastError();
}

template <int D>
cudaError_t attn_bwd_launch_d(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                              const float* lse, float* stats, void* dq, void* dk, void* dv, int B, int T, int H,
                              int Hkv, float scale, int* status, cudaStream_t stream) {
  CUtensorMap qs, dos, ks, vs;
  const uint64_t wq = (uint64_t)H * D, wk = (uint64_t)Hkv * D;
  if (!attn_tmap_seq(&qs, q, wq, T, B) || !attn_tmap_seq(&dos, d_o, wq, T, B) || !attn_tmap_seq(&ks, k, wk, T, B) ||
      !attn_tmap_seq(&vs, v, wk, T, B))
    return cudaErrorInvalidValue;
  auto kq = attn_bwd_dq_kernel<D>;
  auto kkv = attn_bwd_dkv_kernel<D>;
  static std::atomic<unsigned long long> granted{0};
  const cudaError_t e = once_per_device(granted, [&] {
    cudaFuncAttributes fa;
    // the register shares of the kernel's warps add up to what it is launched with, or the larger one waits forever
    if (cudaFuncGetAttributes(&fa, kq) != cudaSuccess || fa.numRegs != 168) return cudaErrorInvalidConfiguration;
    const cudaError_t set = cudaFuncSetAttribute(kq, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdQCfg<D>::SMEM);
    return set != cudaSuccess ? set : cudaFuncSetAttribute(kkv, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdKvCfg<D>::SMEM);
  });
  if (e != cudaSuccess) return e;
  const int tiles = (T + kBM - 1) / kBM, t_pad = tiles * kBM;
  float* neg_lse2 = stats;
  float* neg_delta = stats + (long long)B * H * t_pad;
  const FastDiv by_heads(H);
  constexpr int rows = 256 / (D / 8) * kDeltaRows;  // per block
  if ((t_pad + rows - 1) / rows > 65535) return cudaErrorInvalidValue;
  launch_pdl(attn_delta_kernel<D>, dim3(B * H, (t_pad + rows - 1) / rows), dim3(256), 0, stream, 0,
             reinterpret_cast<const __nv_bfloat16*>(o), reinterpret_cast<const __nv_bfloat16*>(d_o), lse, neg_lse2, neg_delta, T,
             H, t_pad, by_heads, scale);
  const int kv_ctas = attn_grid((long long)B * Hkv * tiles), q_ctas = attn_grid((long long)B * H * tiles);
  AttnBwdParams p;
  p.dq = reinterpret_cast<__nv_bfloat16*>(dq);
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk);
  p.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  p.neg_lse2 = neg_lse2;
  p.neg_delta = neg_delta;
  p.q_plan = WorkPlan(tiles, B * H, q_ctas);
  p.kv_plan = WorkPlan(tiles, B * Hkv, kv_ctas);
  p.by_heads = by_heads;
  p.by_kv_heads = FastDiv(Hkv);
  p.by_group = FastDiv(H / Hkv);
  p.B = B;
  p.T = T;
  p.H = H;
  p.Hkv = Hkv;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  launch_pdl(kkv, dim3(kv_ctas), dim3(kBwdThreads), BwdKvCfg<D>::SMEM, stream, 0, qs, dos, ks, vs, p);
  launch_pdl(kq, dim3(q_ctas), dim3(kDqThreads), BwdQCfg<D>::SMEM, stream, 0, qs, dos, ks, vs, p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t attn_bwd_launch(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                            const float* lse, float* stats, void* dq, void* dk, void* dv, int B, int T, int H, int Hkv,
                            int D, float scale, int* status, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || H <= 0 || Hkv <= 0 || H % Hkv != 0 || B * H > 65535)
    return cudaErrorInvalidValue;
  if (D == 128)
    return attn_bwd_launch_d<128>(q, k, v, o, d_o, lse, stats, dq, dk, dv, B, T, H, Hkv, scale, status, stream);
  if (D == 64)
    return attn_bwd_launch_d<64>(q, k, v, o, d_o, lse, stats, dq, dk, dv, B, T, H, Hkv, scale, status, stream);
  return cudaErrorInvalidValue;
}

cudaError_t attn_fwd_launch(const void* q, const void* k, const void* v, void* out, float* lse, int B, int T, int H,
                            int Hkv, int D, float scale, int* status, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || H <= 0 || Hkv <= 0 || H % Hkv != 0 || B * H > 65535) return cudaErrorInvalidValue;
  if (D == 128) return attn_fwd_launch_d<128>(q, k, v, out, lse, B, T, H, Hkv, scale, status, stream);
  if (D == 64) return attn_fwd_launch_d<64>(q, k, v, out, lse, B, T, H, Hkv, scale, status, stream);
  return cudaErrorInvalidValue;
}

}  // namespace dion
