// All steps of a Newton-Schulz iteration of small matrices in one launch (dion/muon.py:620-647).
//
// A step is three products, each of which needs the whole result of the one before: X X^T, b A + c A A and a X + P X.  For a
// 256 x 256 matrix every one of them is 8 tiles and 0.3 us of multiplying, and as a launch of its own it takes 5 to 6 us.
// Here a cluster of up to eight CTAs takes one matrix and goes through all products with a cluster barrier in between; what
// they hand on passes through the L2.  256 x 256, five steps with the scaling in front: 92 -> 62 us of GPU time.
//
// Everything is multiplied row by row (both operands K-major): the kernel keeps X (k x L, k <= L) and its transpose, A and
// P = b A + c A A are symmetric.  A tile is 128 x 64 so that 256 x 256 gives eight CTAs work, with 24 KB per 64 of K and
// eight such stages: all operands of a tile with K <= 512 are in flight at once.  Warps 0 to 7 write the results of one
// tile while warp 8 loads and warp 9 multiplies the next.  Roundings are those of the products as single launches: bf16
// results of fp32 sums.
//
// Bound by the chain per product, 3.5 us at 256 x 256 (cycles): first load 1600, the other 72 KB into one SM 1550, last MMA to
// epilogue 450, TMEM to shared memory 900 to 1400, stores 200 to 700, barrier with its release 1250.  Results go out by TMA
// because plain stores of rows (16 bytes per lane, 128 apart) took 1200 and the fence between them and the loads 1500.
#include <atomic>

#include "gemm.h"
#include "kernels.h"
#include "pdl.cuh"
#include "per_device.h"
#include "umma.cuh"

namespace dion {
namespace {

typedef __nv_bfloat16 bf16;

constexpr int kTileM = 128, kTileN = 64, kChunk = 64;  // kChunk bf16 of K: the 128 bytes of a swizzled row
constexpr int kStages = 8;
constexpr int kBoxBytes = 64 * kChunk * 2;  // 64 rows
constexpr int kStageBytes = 3 * kBoxBytes;
constexpr int kOutBytes = 2 * kBoxBytes;  // a tile of results, 128 x 64, and the same transposed, 64 x 128: two boxes each
constexpr int kTurnPitch = 72;            // of the input's 64 x 64 tiles: rows of 144 bytes
constexpr int kEpiThreads = 256, kThreads = kEpiThreads + 64;
constexpr int kTmemCols = 2 * kTileN;
constexpr int kMaxSteps = 16;
constexpr int kSmemBytes = kStages * kStageBytes + 2 * kOutBytes + 1024;  // 1024: alignment of the stages
static_assert(2 * kOutBytes >= 64 * kTurnPitch * 2, "the input is transposed in the buffer of the results");

struct NsParams {
  bf16 *X, *A, *Xt[2];
  int k, L, pitch, steps, tall;  // X [k][pitch] (pitch >= L, whole 16 bytes), A [k][k], Xt [L][k]
  int* status;
  float coeffs[3 * kMaxSteps];
};

struct Shared {
  uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
  uint32_t tmem;
  int abort;
};

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// orders this thread's plain accesses to global memory with bulk copies (over all state spaces it takes 650 cycles longer)
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
// every committed bulk store of this thread has reached memory
__device__ __forceinline__ void tma_store_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void give_up(Shared& sh, int* status, int code) {
  *reinterpret_cast<volatile int*>(&sh.abort) = 1;
  if (status) atomicCAS(status, 0, code);
}

// one answer for all lanes of a converged warp
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

struct Product {
  const CUtensorMap *a, *b;  // both [rows][K]
  int tiles_n, tiles, chunks;
};

__global__ void __launch_bounds__(kThreads, 1)
    newton_schulz_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_a,
                         const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_t0,
                         const __grid_constant__ CUtensorMap map_t1, const __grid_constant__ NsParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* stages = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint8_t* const tile_rows = stages + kStages * kStageBytes;
  uint8_t* const tile_cols = tile_rows + kOutBytes;
  __shared__ Shared sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ctas = gridDim.x, rank = blockIdx.x, batch = blockIdx.y;  // a cluster is a row of the grid

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.acc_full[i], 1);
      mbar_init(&sh.acc_empty[i], kEpiThreads / 32);
    }
    sh.abort = 0;
    mbar_fence_init();
  }
  pdl_wait();  // before tensor memory is taken, which a kernel ahead of this one may still be waiting for
  if (warp == 8) {
    tmem_alloc(&sh.tmem, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(sh.tmem);
  volatile int* abort_flag = &sh.abort;

  const int k = p.k, L = p.L, pitch = p.pitch;
  bf16* X = p.X + (long long)batch * k * pitch;
  bf16* A = p.A + (long long)batch * k * k;
  bf16* const Xt[2] = {p.Xt[0] + (long long)batch * L * k, p.Xt[1] + (long long)batch * L * k};

  // the input lies in X, or in Xt[0] when tall: fill the other
  if (warp < 8) {
    bf16* turned = reinterpret_cast<bf16*>(tile_rows);
    const bf16* src = p.tall ? Xt[0] : X;
    bf16* dst = p.tall ? X : Xt[0];
    const int rows = p.tall ? L : k, cols = p.tall ? k : L, sp = p.tall ? k : pitch, dp = p.tall ? pitch : k;
    const int tc = (cols + 63) / 64, count = (rows + 63) / 64 * tc;
    for (int t = rank; t < count; t += ctas) {
      const int r0 = t / tc * 64, c0 = t % tc * 64;
      epi_sync();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int v = threadIdx.x + i * kEpiThreads, r = v >> 3, c = (v & 7) * 8;
        uint4 q = make_uint4(0, 0, 0, 0);
        if (r0 + r < rows && c0 + c < cols) q = *reinterpret_cast<const uint4*>(src + (long long)(r0 + r) * sp + c0 + c);
        const bf16* e = reinterpret_cast<const bf16*>(&q);
#pragma unroll
        for (int j = 0; j < 8; ++j) turned[(c + j) * kTurnPitch + r] = e[j];
      }
      epi_sync();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int v = threadIdx.x + i * kEpiThreads, c = v >> 3, r = (v & 7) * 8;
        // the last vector of a row of X may reach into the padding of its pitch, which is zero and stays so
        if (c0 + c < cols && r0 + r < rows)
          *reinterpret_cast<uint4*>(dst + (long long)(c0 + c) * dp + r0 + r) = *reinterpret_cast<const uint4*>(turned + c * kTurnPitch + r);
      }
    }
    fence_proxy_async_global();
    epi_sync();  // the results' buffer is free
  }
  cluster_sync_all();

  const int tm = (k + kTileM - 1) / kTileM, tk = (k + kTileN - 1) / kTileN, tl = (L + kTileN - 1) / kTileN;
  uint32_t it = 0, tile = 0;  // chunks and tiles so far; every role counts for itself
  bool dead = false;          // of the multiplying warp
  for (int step = 0; step < p.steps; ++step) {
    const int cur = step & 1;
    const bool last = step + 1 == p.steps;
    for (int which = 0; which < 3; ++which) {
      Product g;
      g.a = which == 0 ? &map_x : which == 1 ? &map_a : &map_p;
      g.b = which == 0 ? &map_x : which == 1 ? &map_a : cur ? &map_t1 : &map_t0;
      g.tiles_n = which == 2 ? tl : tk;
      g.tiles = tm * g.tiles_n;
      g.chunks = ((which == 0 ? pitch : k) + kChunk - 1) / kChunk;

      if (warp == 8) {
        if (lane == 0) {
          fence_proxy_async_global();
          for (int t = rank; t < g.tiles && !*abort_flag; t += ctas) {
            const int m0 = t / g.tiles_n * kTileM, n0 = t % g.tiles_n * kTileN;
            for (int c = 0; c < g.chunks; ++c, ++it) {
              const int s = it % kStages;
              if (it >= kStages && !mbar_wait(&sh.empty[s], ((it / kStages) & 1) ^ 1, abort_flag)) {
                give_up(sh, p.status, kStatusProducerTimeout);
                break;
              }
              uint8_t* to = stages + s * kStageBytes;
              mbar_arrive_expect_tx(&sh.full[s], kStageBytes);
              tma_load_3d(to, g.a, &sh.full[s], c * kChunk, m0, batch);
              tma_load_3d(to + kBoxBytes, g.a, &sh.full[s], c * kChunk, m0 + 64, batch);
              tma_load_3d(to + 2 * kBoxBytes, g.b, &sh.full[s], c * kChunk, n0, batch);
            }
          }
        }
      } else if (warp == 9) {
        constexpr uint32_t idesc = make_instr_desc(1, 0, 0, kTileM, kTileN);
        for (int t = rank; t < g.tiles && !dead; t += ctas, ++tile) {
          const uint32_t acc = tile & 1;
          if (tile >= 2) dead = !warp_wait(&sh.acc_empty[acc], ((tile >> 1) & 1) ^ 1, abort_flag);
          for (int c = 0; c < g.chunks && !dead; ++c, ++it) {
            const int s = it % kStages;
            dead = !warp_wait(&sh.full[s], (it / kStages) & 1, abort_flag);
            if (dead) break;
            tc_fence_after();
            const uint32_t at = smem_u32(stages + s * kStageBytes);
            const uint64_t da = make_smem_desc(at, 0, 1024), db = make_smem_desc(at + 2 * kBoxBytes, 0, 1024);
            if (elect_one()) {
#pragma unroll
              for (int j = 0; j < kChunk / 16; ++j)
                umma_ss<false>(tmem + acc * kTileN, da + 2 * j, db + 2 * j, idesc, c > 0 || j > 0);
              umma_commit(&sh.empty[s]);
              if (c + 1 == g.chunks) umma_commit(&sh.acc_full[acc]);
            }
            __syncwarp();
          }
          if (dead) give_up(sh, p.status, kStatusMmaTimeout);
        }
      } else {
        const bool to_rows = which < 2 || !(last && p.tall), to_cols = which == 2 && !(last && !p.tall);
        const float alpha = which == 1 ? p.coeffs[3 * step + 2] : 1.f;
        const float beta = which == 0 ? 0.f : which == 1 ? p.coeffs[3 * step + 1] : p.coeffs[3 * step];
        const bf16* add = which == 1 ? A : X;
        const CUtensorMap* out_rows = which == 0 ? &map_a : which == 1 ? &map_p : &map_x;
        const CUtensorMap* out_cols = cur ? &map_t0 : &map_t1;
        const int ld = which == 2 ? pitch : k;
        for (int t = rank; t < g.tiles; t += ctas, ++tile) {
          const uint32_t acc = tile & 1;
          const int row = t / g.tiles_n * kTileM + (warp & 3) * 32 + lane;
          const int half = (warp >> 2) * 32, col0 = t % g.tiles_n * kTileN + half;  // this thread: 32 columns of a row
          const long long at = (long long)row * ld + col0;
          uint4 addend[4];
          if (which > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (row < k && col0 + 8 * i < ld) addend[i] = __ldcg(reinterpret_cast<const uint4*>(add + at) + i);
          }
          // a warp whose wait ran out goes on through the barriers, with whatever the accumulator holds
          if (!warp_wait(&sh.acc_full[acc], (tile >> 1) & 1, abort_flag)) give_up(sh, p.status, kStatusEpilogueTimeout);
          tc_fence_after();
          float v[32];
          tmem_ld_32x32(tmem + acc * kTileN + half + ((uint32_t)((warp & 3) * 32) << 16), v);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.acc_empty[acc]);
          if (which > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&addend[i]);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(e[j]);
                v[8 * i + 2 * j] = alpha * v[8 * i + 2 * j] + beta * f.x;
                v[8 * i + 2 * j + 1] = alpha * v[8 * i + 2 * j + 1] + beta * f.y;
              }
            }
          }
          uint4 q[4];
#pragma unroll
          for (int i = 0; i < 16; ++i)
            reinterpret_cast<__nv_bfloat162*>(q)[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
          // the tile as TMA stores read it: 64 columns in 128-byte rows, 16-byte units swizzled by the row
          const int m0 = t / g.tiles_n * kTileM, n0 = t % g.tiles_n * kTileN, r = (warp & 3) * 32 + lane;
          if (t != rank) {
            if (threadIdx.x == 0) tma_store_wait_read();
            epi_sync();
          }
          if (to_rows) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(tile_rows + r * 128 + (((half >> 3) + i) ^ (r & 7)) * 16) = q[i];
          }
          if (to_cols) {
            const bf16* e = reinterpret_cast<const bf16*>(q);
            uint8_t* box = tile_cols + (r >> 6) * kBoxBytes + (r & 7) * 2;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              *reinterpret_cast<bf16*>(box + (half + j) * 128 + ((((r & 63) >> 3) ^ (j & 7)) * 16)) = e[j];
          }
          fence_proxy_async_shared();
          epi_sync();
          if (threadIdx.x == 0) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (to_rows && m0 + 64 * i < k) tma_store_3d(out_rows, tile_rows + i * kBoxBytes, n0, m0 + 64 * i, batch);
              if (to_cols && m0 + 64 * i < k) tma_store_3d(out_cols, tile_cols + i * kBoxBytes, m0 + 64 * i, n0, batch);
            }
            tma_store_commit();
          }
        }
        if (threadIdx.x == 0) tma_store_wait();  // a completed bulk store is seen by plain loads as well (the addends)
      }
      // Also when a wait ran out: nobody is left waiting.  Only the thread that stored the tiles has something to release.
      __syncwarp();
      if (!(last && which == 2)) {
        if (warp == 0) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      }
    }
  }
  // copies still in flight after a wait ran out
  if (warp == 8 && lane == 0 && *abort_flag) {
    int again = 0;
    for (uint32_t i = it > kStages ? it - kStages : 0; i < it; ++i) mbar_wait(&sh.full[i % kStages], (i / kStages) & 1, &again);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 8) tmem_dealloc(tmem, kTmemCols);
}

int tiles_of(int rows, int cols) { return (rows + kTileM - 1) / kTileM * ((cols + kTileN - 1) / kTileN); }

// CTAs per matrix: as many as have a tile each, if all clusters run at once on the SMs of a B200 (one CTA per SM; 12 clusters
// of eight, 24 of four and 64 of two do, 16, 36 and 128 do not: 16 x 256 x 256 63 -> 118 us), 0 if no size does.
int cluster_size(int batch, int k, int L) {
  const int room = batch <= 12 ? 8 : batch <= 24 ? 4 : batch <= 64 ? 2 : batch <= 128 ? 1 : 0;
  int c = 1;
  while (c < room && c < tiles_of(k, L)) c *= 2;
  return room == 0 ? 0 : c;
}

}  // namespace

// What a CTA does one after the other in a step, in loads of 24 KB (0.28 us; another tile costs two): up to 22 of them and
// the three hand-overs take less than three launches.  Five steps as launches and here, us (the loads in brackets):
//   1 x 64 x 64 72 / 44 (3), 64 x 64 x 64 73 / 47 (3), 1 x 128 x 128 74 / 52 (6), 36 x 128 x 256 85 / 70 (12),
//   128 x 128 x 128 91 / 86 (18), 1 x 192 x 512 89 / 74 (19), 1 x 256 x 256 92 / 62 (12), 12 x 256 x 512 108 / 83 (22),
// and beyond: 16 x 192 x 192 90 / 81 (24), 36 x 128 x 512 92 / 101 (24), 16 x 256 x 256 101 / 94 (30),
//   1 x 256 x 768 101 / 101 (32), 1 x 64 x 2048 94 / 110 (39), 1 x 256 x 1024 104 / 119 (42).
bool newton_schulz_takes(long long batch, long long k, long long L, int steps) {
  if (batch < 1 || batch > 128 || k < 8 || k % 8 != 0 || k > 256 || L < k || L > 1536 || steps < 1 || steps > kMaxSteps) return false;
  const int c = cluster_size((int)batch, (int)k, (int)L);
  if (c == 0) return false;
  const int square = (tiles_of((int)k, (int)k) + c - 1) / c, wide = (tiles_of((int)k, (int)L) + c - 1) / c;  // tiles per CTA
  const int kc = ((int)k + kChunk - 1) / kChunk, lc = ((int)L + kChunk - 1) / kChunk;
  return (lc + kc) * square + kc * wide + 2 * (2 * square + wide - 3) <= 22;
}

cudaError_t newton_schulz_launch(void* X, void* A, void* P, void* Xt0, void* Xt1, int batch, int k, int L, int pitch,
                                 const float* coeffs, int steps, bool tall, int* status, cudaStream_t stream) {
  if (steps < 1 || steps > kMaxSteps || k % 8 != 0 || pitch % 8 != 0 || pitch < L) return cudaErrorInvalidValue;
  CUtensorMap mx, ma, mp, m0, m1;
  if (!bf16_tile_map(&mx, X, pitch, k, batch, pitch, (uint64_t)k * pitch, kChunk, 64) ||
      !bf16_tile_map(&ma, A, k, k, batch, k, (uint64_t)k * k, kChunk, 64) ||
      !bf16_tile_map(&mp, P, k, k, batch, k, (uint64_t)k * k, kChunk, 64) ||
      !bf16_tile_map(&m0, Xt0, k, L, batch, k, (uint64_t)L * k, kChunk, 64) ||
      !bf16_tile_map(&m1, Xt1, k, L, batch, k, (uint64_t)L * k, kChunk, 64))
    return cudaErrorInvalidValue;
  NsParams p;
  p.X = (bf16*)X, p.A = (bf16*)A, p.Xt[0] = (bf16*)Xt0, p.Xt[1] = (bf16*)Xt1;
  p.k = k, p.L = L, p.pitch = pitch, p.steps = steps, p.tall = tall, p.status = status;
  for (int i = 0; i < 3 * kMaxSteps; ++i) p.coeffs[i] = i < 3 * steps ? coeffs[i] : 0.f;
  static std::atomic<unsigned long long> granted{0};
  const cudaError_t e = once_per_device(
      granted, [] { return cudaFuncSetAttribute(newton_schulz_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes); });
  if (e != cudaSuccess) return e;
  const unsigned c = cluster_size(batch, k, L);
  if (c == 0) return cudaErrorInvalidValue;
  return launch_pdl(newton_schulz_kernel, dim3(c, batch), dim3(kThreads), kSmemBytes, stream, c, mx, ma, mp, m0, m1, p);
}

}  // namespace dion
