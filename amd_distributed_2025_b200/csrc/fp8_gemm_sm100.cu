// Block-scaled fp8 (e4m3) GEMM for sm_100a:  C[m, n] = sum_kb (A_kb[m, :] . B_kb[n, :]) * as[m, kb] * bs[n / 128, kb]
//
// The reference tree carries a template for this operation that belongs to neither of
// its two tasks (all2all/hip.py:17-59, identical copy in gemm-rs/hip.py): one thread per
// output element, K walked in blocks of 128, the block's partial product multiplied by a
// per-row scale of A and a per-128x128-block scale of B, bf16 result.  Here the block
// products run on the tensor cores.  Operands are K-major (row-major [m, k] and [n, k]); TMA stages
// them with the 128-byte swizzle exactly as in the bf16 GEMM (a 128-byte row now holds 128 fp8 values).
//
// A CTA pair (cta_group::2) owns a tile of 256 rows of A by 64, 128, 192 or 256 rows of B.  Every 128-wide K block is
// multiplied into tensor memory of its own, in one of two buffers (two neighbouring blocks to a buffer where the tile has
// at most 128 columns); eight epilogue warps, two per tensor-memory lane quarter, pull the products out, multiply by
// the blocks' scales and accumulate in fp32 registers while the next buffer is being filled.  Two warps bring the scales
// in by asynchronous copies, sixteen blocks ahead: a row's scales lie in a line of their own, and fetched by the
// epilogue itself they took longer than the products.  A warp of a 256-column tile holds 128 sums and 64 products a lane,
// so registers are split: 232 for the epilogue, 40 for the others.  Pairs are persistent; where there are fewer tiles
// than pairs, a cluster of pairs shares a tile (of up to 128 columns), each over its part of K, and the parts meet in
// distributed shared memory.
//
// What bounds it, in cycles per K block: tiles of up to 128 columns the operands (192 rows for 128 columns: 500 without
// the epilogue, where the products alone take 300); wider ones the chain of one epilogue warp.  By its own clock, at
// 4096 x 4096 x 2048 on tiles of 256 columns: 1000 cycles a K block, where the products alone take 560 -- 150 waiting for
// the products, 320 for two reads with 64 packed additions each, 55 for the signal that frees the buffer, 200 for the
// scales of the next step, and 275 between the stamps that have no name -- and 2480 a tile, 2030 of them the result's way
// out: four waves of 18500 cycles are the 37.7 us that it takes cool.  So the chain is kept short: one lane signals by
// predicate, not by branch; the wide tile fetches its next scales before it adds.  In a long row of calls the clock goes
// down to 1700 MHz (42 us), and wide tiles move a third less operand data.
// On a B200, us, cool / in a row of calls, tiles of up to 128 columns with branches -> now:
//   4096 x 4096 x 2048 38.1 / 45.8 -> 37.2 / 43.5   8192 x 8192 x 4096 268 / 310 -> 241 / 281   2048^3 13.4 -> 12.4
//   3545 x 4512 x 3824 78.5 / 90.5 -> 65 / 76       2048 x 5000 x 8192 84 / 102 -> 79 / 95
//   1024 x 4096 x 4096 21.1 -> 19.7
// Tried and slower: sixteen epilogue warps (52 us at 4096 x 4096 x 2048, the waits doubled), warp-wide waits (40.8), chunks
// read one by one (47.5), results by 32-byte stores (44.8), the last wave's tiles in halves for twice the pairs (level).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "fp8_gemm.h"
#include "gemm_rs.h"
#include "per_device.h"
#include "plan_cache.h"
#include "signal.cuh"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace b200 {

namespace {

constexpr int kRows = 128;                // rows of A per CTA
constexpr int kBlockK = 128;              // the scale block of the operation: one 128-byte row
constexpr int kABytes = kRows * kBlockK;
constexpr int kEpiWarps = 8;
constexpr int kScaleWarps = 2;
constexpr int kThreads = 64 + 32 * (kScaleWarps + kEpiWarps);
// Registers per thread: the epilogue's two warpgroups take what the first one (copies, products, scales) gives up.
constexpr int kLightRegs = 40, kEpiRegs = 232;
static_assert(128 * kLightRegs + 256 * kEpiRegs == kThreads * 168, "not more than the block is launched with");
constexpr int kMaxStages = 12;
constexpr int kSlabBytes = 2 * 2048;      // per epilogue warp: two buffers of 32 rows x 64 bytes
constexpr int kMaxChunks = 4;             // 32-column chunks of an epilogue warp
constexpr int kGroup = 4;                 // K blocks whose scales come in together
constexpr int kScaleSlots = 4;
constexpr int kScaleBytes = kGroup * (kRows + 2 * kMaxChunks) * 4;  // [row][block], then [block][half of the columns][chunk]
constexpr int kTailBytes = kEpiWarps * kSlabBytes + kScaleSlots * kScaleBytes + 512;
constexpr int kBufs = 2;                  // tensor-memory buffers of 256 columns
constexpr int kMaxDynamicSmem = 232448 - 256;
constexpr int kTmemCols = 512;

struct Fp8Params {
  const float* a_scale;  // [m, k_blocks], element (m, kb) at m * as_stride_m + kb * as_stride_k
  const float* b_scale;  // [n_blocks, k_blocks], element (nb, kb) at nb * bs_stride_n + kb * bs_stride_k
  __nv_bfloat16* c;      // [m, n] row-major
  int M, N, k_blocks;
  long long as_stride_m, as_stride_k, bs_stride_n, bs_stride_k;
  int m_tiles, n_tiles, band, stages, stage_area;
  int splits;            // pairs of a cluster that share a tile
  int tma_out;           // 1: rows of C are whole 16-byte pieces: results leave through TMA
  uint64_t timeout_ns;   // of a pipeline wait
  StatusWord* status;    // mapped host memory
};

// Instruction descriptor of tcgen05.mma.kind::f8f6f4 with e4m3 A and B (both K-major) and fp32
// accumulation: bits [4,6) D format (1 = f32), [7,10) A format (0 = e4m3), [10,13) B format,
// [17,23) N >> 3, [24,29) M >> 4.
__device__ __forceinline__ uint32_t make_idesc_e4m3_f32(int m, int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void umma_fp8_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// `detail` (not 0) tells which wait it was that expired: a hundred for the kind of barrier, plus its index.
__device__ __forceinline__ bool fp8_wait(uint32_t bar, uint32_t parity, volatile int* abort, const Fp8Params& p,
                                         int detail) {
  uint64_t t0 = 0;  // (the clock takes longer to read than most waits last)
  for (uint32_t spins = 1; !ptx::mbar_try_wait(bar, parity); ++spins) {
    if ((spins & 255u) == 0) {
      if (*abort) return false;
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > p.timeout_ns) {
        *abort = detail;
        return false;
      }
    }
  }
  return true;
}

// A CTA in which a wait expired says so on its way out (every warp that knows of it does, and one is enough): what it
// computed is of no use.
__device__ __forceinline__ void record_expired(const Fp8Params& p, int detail) {
  if (p.status != nullptr && reinterpret_cast<volatile StatusWord*>(p.status)->code == STATUS_OK)
    store_status(p.status, STATUS_TIMEOUT, PHASE_GEMM_PIPELINE, -1, detail, 0, 0);
}

// acc[0..1] += v[0..1] * s
__device__ __forceinline__ void fma2(float2& acc, uint32_t v0, uint32_t v1, float2 ss) {
  const float2 v = make_float2(__uint_as_float(v0), __uint_as_float(v1));
  // (volatile: not before the wait for the tensor memory load that brings v)
  asm volatile("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(acc))
      : "l"(reinterpret_cast<const unsigned long long&>(v)), "l"(reinterpret_cast<const unsigned long long&>(ss)));
}

template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t to, const float* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(from), "n"(BYTES) : "memory");
}

// Arrives on `bar` when this thread's copies so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void ld_shared_f4(float* to, uint32_t from) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(to[0]), "=f"(to[1]), "=f"(to[2]), "=f"(to[3])
               : "r"(from)
               : "memory");
}

__device__ __forceinline__ uint32_t pack2(float2 f) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

}  // namespace

// CHUNKS: 32-column chunks of an epilogue warp; the tile has 64 * CHUNKS columns.
template <int CHUNKS>
__global__ void __launch_bounds__(kThreads, 1)
fp8_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ CUtensorMap map_c, const Fp8Params p) {
  constexpr int kBn = 64 * CHUNKS;
  constexpr int kStep = CHUNKS <= 2 ? 2 : 1;  // K blocks to a tensor-memory buffer
  constexpr bool kAhead = CHUNKS == 4;
  constexpr bool kShared = CHUNKS <= 2;       // tiles that a cluster of pairs may share
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int abort_flag;
  __shared__ uint32_t tmem_base_shared;

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int splits = kShared ? p.splits : 1;
  const int cluster_rank = (int)ptx::cluster_ctarank();
  const int rank = cluster_rank >> 1;  // which part of K
  const int cta = cluster_rank & 1;    // which half of the pair's rows
  // parts of K; even bounds where that is little of a part, so that scales still come in by pieces of 8 bytes
  const int round = p.k_blocks >= 4 * splits ? ~1 : ~0;
  const int kb0 = (int)((int64_t)p.k_blocks * rank / splits) & round;
  const int kb1 = rank + 1 == splits ? p.k_blocks : (int)((int64_t)p.k_blocks * (rank + 1) / splits) & round;
  const int first_tile = (int)blockIdx.x / (2 * splits);
  const int tile_step = (int)gridDim.x / (2 * splits);
  const int total = p.m_tiles * p.n_tiles;
  constexpr int b_rows = kBn / 2;  // rows of B that this CTA brings in
  constexpr uint32_t buf_cols = kTmemCols / kBufs;
  constexpr uint32_t block_cols = buf_cols / kStep;

  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t stage_bytes = kABytes + (uint32_t)b_rows * kBlockK;
  const uint32_t slabs = base + (uint32_t)p.stage_area;
  const uint32_t scales = slabs + kEpiWarps * kSlabBytes;
  const uint32_t bars = scales + kScaleSlots * kScaleBytes;
  auto full_bar = [&](uint32_t s) { return bars + 8u * s; };
  auto empty_bar = [&](uint32_t s) { return bars + 8u * (kMaxStages + s); };
  auto tfull_bar = [&](uint32_t s) { return bars + 8u * (2 * kMaxStages + s); };
  auto tempty_bar = [&](uint32_t s) { return bars + 8u * (2 * kMaxStages + kBufs + s); };
  auto sfull_bar = [&](uint32_t s) { return bars + 8u * (2 * kMaxStages + 2 * kBufs + s); };
  auto sempty_bar = [&](uint32_t s) { return bars + 8u * (2 * kMaxStages + 2 * kBufs + kScaleSlots + s); };

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < kBufs; ++s) {
      ptx::mbar_init(tfull_bar(s), 1);
      ptx::mbar_init(tempty_bar(s), 2 * kEpiWarps);
    }
    for (int s = 0; s < kScaleSlots; ++s) {
      ptx::mbar_init(sfull_bar(s), 32 * kScaleWarps);
      ptx::mbar_init(sempty_bar(s), kEpiWarps);
    }
    ptx::fence_mbar_init();
    ptx::fence_proxy_async_smem();
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
    ptx::prefetch_tensormap(&map_c);
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(ptx::smem_u32(&tmem_base_shared), kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_shared;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();

  // bands of row tiles, column tile by column tile: pairs at work at the same time share operands in L2
  auto tile_coords = [&](int tile, int& mt, int& nt) {
    const int per_band = p.band * p.n_tiles;
    const int b = tile / per_band;
    const int start = b * p.band;
    const int size = min(p.band, p.m_tiles - start);
    const int within = tile - start * p.n_tiles;
    nt = within / size;
    mt = start + within - nt * size;
  };

  // All of a CTA's threads come here in the end, each role on its own way: no CTA retires while another may still signal
  // its barriers or read its memory.
  auto leave = [&]() {
    if (abort_flag) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
      if (lane == 0) record_expired(p, abort_flag);
    }
    __syncwarp();
    ptx::tcgen05_fence_before();
    __syncthreads();
    ptx::cluster_sync_all();
    ptx::tcgen05_fence_after();
    if (warp == 1) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
  };

  if (warp < 2 + kScaleWarps) {
    ptx::setmaxnreg_dec<kLightRegs>();
    if (warp == 0) {
      uint32_t stage = 0, phase = 0;
      for (int tile = first_tile; tile < total && !abort_flag; tile += tile_step) {
        int mt, nt;
        tile_coords(tile, mt, nt);
        const int ay = mt * 256 + cta * kRows;
        const int by = nt * kBn + cta * b_rows;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!fp8_wait(empty_bar(stage), phase ^ 1u, &abort_flag, p, 100 + (int)stage)) break;
          const uint32_t sa = base + stage * stage_bytes;
          if (ptx::elect_one()) {
            if (cta == 0) ptx::mbar_arrive_expect_tx(full_bar(stage), 2 * stage_bytes);
            ptx::tma_load_2d_pair(sa, &map_a, full_bar(stage), kb * kBlockK, ay);
            ptx::tma_load_2d_pair(sa + kABytes, &map_b, full_bar(stage), kb * kBlockK, by);
          }
          __syncwarp();
          if (++stage == (uint32_t)p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    } else if (warp == 1) {
      if (cta == 0) {
        const uint32_t idesc = make_idesc_e4m3_f32(256, kBn);
        const uint16_t both = (uint16_t)(3u << (2 * rank));
        uint32_t stage = 0, phase = 0, buf = 0, buf_phase = 0;
        for (int tile = first_tile; tile < total && !abort_flag; tile += tile_step) {
          bool ok = true;
          for (int kb = kb0; kb < kb1 && ok; kb += kStep) {
            ok = fp8_wait(tempty_bar(buf), buf_phase ^ 1u, &abort_flag, p, 200 + (int)buf);
            ptx::tcgen05_fence_after();
#pragma unroll
            for (int i = 0; i < kStep; ++i) {
              if (kb + i >= kb1) break;
              ok = ok && fp8_wait(full_bar(stage), phase, &abort_flag, p, 300 + (int)stage);
              if (!ok) break;
              ptx::tcgen05_fence_after();
              const uint32_t sa = base + stage * stage_bytes;
              const uint64_t da = ptx::make_smem_desc_k_sw128(sa);
              const uint64_t db = ptx::make_smem_desc_k_sw128(sa + kABytes);
              const uint32_t d = tmem_base + buf * buf_cols + i * block_cols;
              if (ptx::elect_one()) {
#pragma unroll
                for (int j = 0; j < kBlockK / 32; ++j)  // 32 fp8 of K = 32 bytes = 2 descriptor address units
                  umma_fp8_pair(d, da + 2u * j, db + 2u * j, idesc, j > 0 ? 1u : 0u);
                ptx::umma_commit_pair(empty_bar(stage), both);
                if (i == kStep - 1 || kb + i + 1 == kb1) ptx::umma_commit_pair(tfull_bar(buf), both);
              }
              __syncwarp();
              if (++stage == (uint32_t)p.stages) {
                stage = 0;
                phase ^= 1u;
              }
            }
            if (++buf == (uint32_t)kBufs) {
              buf = 0;
              buf_phase ^= 1u;
            }
          }
          if (!ok) break;
        }
      }
    } else {
      // ---- scales: two rows per lane, four K blocks at a time, sixteen under way ------------------------------
      const int l = (warp - 2) * 32 + lane;
      // how many neighbouring scales of a row one copy may take: addresses, group starts and the end of the row allow it
      const uint64_t ends =
          reinterpret_cast<uintptr_t>(p.a_scale) / 4 | (uint64_t)p.as_stride_m | (uint64_t)kb0 | (uint64_t)p.k_blocks;
      const int wide = p.as_stride_k != 1 || ends % 2 != 0 ? 1 : ends % 4 != 0 ? 2 : 4;
      uint32_t slot = 0, phase = 0;
      for (int tile = first_tile; tile < total && !abort_flag; tile += tile_step) {
        int mt, nt;
        tile_coords(tile, mt, nt);
        const int m0 = mt * 256 + cta * kRows;
        for (int kb = kb0; kb < kb1; kb += kGroup) {
          if (!fp8_wait(sempty_bar(slot), phase ^ 1u, &abort_flag, p, 500 + (int)slot)) break;
          const uint32_t at = scales + slot * kScaleBytes;
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int row = l + 64 * r;
            if (m0 + row >= p.M) break;  // (nobody reads what such a row multiplies)
            const float* as = p.a_scale + (long long)(m0 + row) * p.as_stride_m;
            const uint32_t to = at + (uint32_t)row * 16u;
            if (wide == 4) {  // (kb + 3 < k_blocks)
              cp_async<16>(to, as + kb);
            } else if (wide == 2) {
              cp_async<8>(to, as + kb);
              cp_async<8>(to + 8u, as + min(kb + 2, p.k_blocks - 2));
            } else {
#pragma unroll
              for (int i = 0; i < kGroup; ++i)
                cp_async<4>(to + 4u * i, as + (long long)min(kb + i, p.k_blocks - 1) * p.as_stride_k);
            }
          }
          if (l < 2 * kMaxChunks * kGroup) {  // block l / 8, chunk l % 8: the first half's in words 0.., the second's in 4..
            const int chunk = (l & 4 ? CHUNKS : 0) + (l & 3);
            const int n = min(nt * kBn + chunk * 32, p.N - 1);
            const int block = min(kb + (l >> 3), p.k_blocks - 1);
            cp_async<4>(at + (uint32_t)(kGroup * kRows + l) * 4u,
                        p.b_scale + (long long)(n >> 7) * p.bs_stride_n + (long long)block * p.bs_stride_k);
          }
          cp_async_arrive(sfull_bar(slot));
          if (++slot == kScaleSlots) {
            slot = 0;
            phase ^= 1u;
          }
        }
      }
    }
    if (splits > 1) {
      __syncwarp();
      ptx::cluster_sync_all();
      ptx::cluster_sync_all();
    }
    leave();
    return;
  }

  // ---- epilogue: two warps per tensor-memory lane quarter, each for half of the columns ---------------------
  ptx::setmaxnreg_inc<kEpiRegs>();
  const int ew = warp - 2 - kScaleWarps;
  const int q = warp & 3;
  const int half = ew >> 2;
  float2 acc[CHUNKS][16];  // this lane's row
  bool alive = true;
  {
    const uint32_t slab = slabs + (uint32_t)ew * kSlabBytes;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * CHUNKS * 32);
    const uint32_t leader_tempty = ptx::map_cluster(tempty_bar(0), (uint32_t)(2 * rank));  // on the pair's leader
    uint32_t buf = 0, buf_phase = 0, slot = 0, slot_phase = 0;
    for (int tile = first_tile; tile < total && !abort_flag; tile += tile_step) {
      int mt, nt;
      tile_coords(tile, mt, nt);
      const int row0 = mt * 256 + cta * kRows + q * 32;
      const int n0 = nt * kBn + half * CHUNKS * 32;
      const int m = row0 + lane;
      const bool rows_in = row0 < p.M;
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[i][j] = make_float2(0.f, 0.f);
      // Scales come out of shared memory a step ahead: a lane's for its row and four K blocks at once, the columns' block by
      // block.  (Where a wait expires, the numbers are of no use any more; the loops still end, and `alive` is asked after
      // them.)
      int g = 0;  // which of the K blocks whose scales came in together
      float sa[kGroup], sb[kStep][4];
      const uint32_t row_at = scales + (uint32_t)(q * 32 + lane) * 16u;
      const uint32_t column_at = scales + (uint32_t)(kGroup * kRows + half * kMaxChunks) * 4u;
      auto fetch_rows = [&]() {
        alive &= fp8_wait(sfull_bar(slot), slot_phase, &abort_flag, p, 600 + (int)slot);
        __syncwarp();
        ld_shared_f4(sa, row_at + slot * kScaleBytes);
      };
      auto fetch_columns = [&]() {
#pragma unroll
        for (int i = 0; i < kStep; ++i)
          ld_shared_f4(sb[i], column_at + slot * kScaleBytes + (uint32_t)((g + i) * 2 * kMaxChunks * 4));
      };
      auto next_step = [&](bool more) {
        g += kStep;
        if (g == kGroup || !more) {
          g = 0;
          __syncwarp();
          ptx::mbar_arrive_if(lane == 0, sempty_bar(slot));
          if (++slot == kScaleSlots) {
            slot = 0;
            slot_phase ^= 1u;
          }
          if (more) fetch_rows();
        }
        if (more) fetch_columns();
      };
      fetch_rows();
      fetch_columns();
#pragma unroll 1
      for (int kb = kb0; kb < kb1; kb += kStep) {
        alive &= fp8_wait(tfull_bar(buf), buf_phase, &abort_flag, p, 400 + (int)buf);
        __syncwarp();
        ptx::tcgen05_fence_after();
        const bool more = kb + kStep < kb1;
        auto done = [&]() {  // the buffer is free for the next products (the warp is converged, and its reads are complete)
          ptx::tcgen05_fence_before();
          ptx::mbar_arrive_remote_if(lane == 0, leader_tempty + 8u * buf);
        };
        if (!rows_in) {
          done();
          next_step(more);
        } else {
          constexpr int kChunks = CHUNKS * kStep;  // of the buffer, block by block, two at a time
          const int here = kStep == 1 || kb + 1 < kb1 ? kChunks : CHUNKS;
          float s[kStep][CHUNKS];
#pragma unroll
          for (int c = 0; c < kChunks; c += 2) {
            if (c < here) {
              uint32_t v[2][32];
#pragma unroll
              for (int d = 0; d < 2; ++d)
                if (c + d < kChunks)
                  ptx::tmem_ld_32x32b_x32(
                      lane_addr + buf * buf_cols + (c + d) / CHUNKS * block_cols + (c + d) % CHUNKS * 32, v[d]);
              if (c == 0) {
#pragma unroll
                for (int i = 0; i < kStep; ++i)
#pragma unroll
                  for (int x = 0; x < CHUNKS; ++x) s[i][x] = sa[i] * sb[i][x];
#pragma unroll
                for (int i = 0; i + kStep < kGroup; ++i) sa[i] = sa[i + kStep];
              }
              ptx::tmem_ld_wait();
              if (c + 2 >= here) {
                done();
                if (kAhead) next_step(more);
              }
#pragma unroll
              for (int d = 0; d < 2; ++d) {
                if (c + d < kChunks && (CHUNKS > 1 || c + d < here)) {
                  const int i = (c + d) / CHUNKS, x = (c + d) % CHUNKS;
#pragma unroll
                  for (int j = 0; j < 16; ++j) fma2(acc[x][j], v[d][2 * j], v[d][2 * j + 1], make_float2(s[i][x], s[i][x]));
                }
              }
            }
          }
        }
        if (!kAhead && rows_in) next_step(more);
        if (++buf == (uint32_t)kBufs) {
          buf = 0;
          buf_phase ^= 1u;
        }
      }
      alive = __all_sync(0xffffffffu, alive);
      if (!alive) break;
      if (!rows_in || splits > 1) continue;
      // ---- result: rounded, through the slab by TMA, or element by element where rows are ragged ------------
      if (p.tma_out) {
#pragma unroll
        for (int i0 = 0; i0 < CHUNKS; i0 += 2) {  // two chunks at a time, a buffer each
          if (lane == 0) ptx::bulk_wait_group_read<0>();  // the stores that used them have read them
          __syncwarp();
#pragma unroll
          for (int i = i0; i < i0 + 2 && i < CHUNKS; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // 16-byte piece j of row `lane`, at the place the 64-byte swizzle wants it
              const uint32_t at = slab + (uint32_t)(i - i0) * 2048u + (uint32_t)lane * 64u +
                                  (uint32_t)((j ^ ((lane >> 1) & 3)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(pack2(acc[i][4 * j])),
                           "r"(pack2(acc[i][4 * j + 1])), "r"(pack2(acc[i][4 * j + 2])), "r"(pack2(acc[i][4 * j + 3]))
                           : "memory");
            }
          }
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
#pragma unroll
            for (int i = i0; i < i0 + 2 && i < CHUNKS; ++i)
              if (n0 + i * 32 < p.N) ptx::tma_store_2d(&map_c, slab + (uint32_t)(i - i0) * 2048u, n0 + i * 32, row0);
            ptx::bulk_commit_group();
          }
        }
      } else if (m < p.M) {
        __nv_bfloat16* row = p.c + (size_t)m * p.N;
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) {
          const int n = n0 + i * 32;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (n + 2 * j < p.N) row[n + 2 * j] = __float2bfloat16_rn(acc[i][j].x);
            if (n + 2 * j + 1 < p.N) row[n + 2 * j + 1] = __float2bfloat16_rn(acc[i][j].y);
          }
        }
      }
    }
    if (lane == 0) ptx::bulk_wait_group_read<0>();
  }

  if (splits > 1) {
    // One tile per cluster.  Columns [r * per, (r + 1) * per) are finished by member r; its pipeline memory, no longer in
    // use anywhere in the cluster after the first barrier, holds [member][per / 4][128 rows] float4.
    int mt, nt;
    tile_coords(first_tile, mt, nt);
    const int row0 = mt * 256 + cta * kRows + q * 32;
    const int per = ((kBn / 8 + splits - 1) / splits) * 8;
    __syncwarp();
    ptx::cluster_sync_all();
    if (alive && row0 < p.M) {
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int col = (half * CHUNKS + i) * 32 + j * 8;
          const int owner = col / per;
          const uint32_t to = (uint32_t)(2 * owner + cta);
          const uint32_t at = base + (uint32_t)((rank * (per / 4) + (col - owner * per) / 4) * kRows + q * 32 + lane) * 16u;
          const float2* a = &acc[i][4 * j];
          ptx::st_cluster_v4(at, to, a[0].x, a[0].y, a[1].x, a[1].y);
          ptx::st_cluster_v4(at + kRows * 16u, to, a[2].x, a[2].y, a[3].x, a[3].y);
        }
      }
    }
    __syncwarp();
    ptx::cluster_sync_all();
    const int m = row0 + lane;
    if (alive && m < p.M) {
      const int c_lo = rank * per;
      const int c_hi = min(kBn, c_lo + per);
      for (int col = c_lo + half * 8; col < c_hi; col += 16) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = 0.f;
        for (int r = 0; r < splits; ++r) {  // ascending k
          const uint32_t from = base + (uint32_t)((r * (per / 4) + (col - c_lo) / 4) * kRows + q * 32 + lane) * 16u;
          float f[8];
          ld_shared_f4(f, from);
          ld_shared_f4(f + 4, from + kRows * 16u);
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] += f[e];
        }
        const int n = nt * kBn + col;
        if (p.tma_out) {  // (rows of whole 16-byte pieces: all eight or none)
          if (n < p.N)
            *reinterpret_cast<uint4*>(p.c + (size_t)m * p.N + n) =
                make_uint4(pack2(make_float2(v[0], v[1])), pack2(make_float2(v[2], v[3])), pack2(make_float2(v[4], v[5])),
                           pack2(make_float2(v[6], v[7])));
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (n + e < p.N) p.c[(size_t)m * p.N + n + e] = __float2bfloat16_rn(v[e]);
        }
      }
    }
  }
  leave();
}

__global__ void fp8_wait_selftest_kernel(const Fp8Params p) {
  __shared__ volatile int abort_flag;
  __shared__ alignas(8) uint64_t bar;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    ptx::mbar_init(ptx::smem_u32(&bar), 1);
    ptx::fence_mbar_init();
  }
  __syncthreads();
  fp8_wait(ptx::smem_u32(&bar), 0, &abort_flag, p, 900);  // nobody arrives
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) record_expired(p, abort_flag);
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
namespace {

struct Fp8Plan {
  int bn = 128, splits = 1, clusters = 1;
  double ns = 1e300;
};

struct Fp8Memory {
  int stages, stage_area;  // multiples of 1024
};
Fp8Memory fp8_memory(int bn, int splits) {
  const int stage_bytes = kABytes + bn / 2 * kBlockK;
  const int parts = splits > 1 ? splits * ((bn / 8 + splits - 1) / splits) * 8 * kRows * 4 : 0;
  Fp8Memory m;
  m.stages = std::min(kMaxStages, (kMaxDynamicSmem - 1024 - kTailBytes) / stage_bytes);
  m.stage_area = std::max(m.stages * stage_bytes, parts);
  return m;
}

// Time model in ns, fitted to 480 timed plans of 120 drawn sizes (0.6 % from the best width of each, with 910 ns in the last
// term throughout; the 450 are from rows of calls and came later): a K block of a tile takes its pair `kb_ns` whatever
// limits it; then power, memory, and what a launch costs before and after its blocks.  A launch that leaves half of the SMs
// idle is set up beside the one before it, which shows most where there is one row of tiles (57 x 4640 x 752: 74 CTAs
// 5.5 us in a row of calls, 146 6.1; but 3409 x 328 x 336: 56 CTAs 6.4, 84 5.5).
Fp8Plan make_fp8_plan(int M, int N, int K, int sms) {
  const int k_blocks = (K + kBlockK - 1) / kBlockK;
  const double dram_ns = ((double)M * K + (double)N * K + 2.0 * M * N) / 6600.0;
  Fp8Plan best;
  for (int bn : {64, 128, 192, 256}) {
    const double kb_ns = bn == 64 ? 230.0 : bn == 128 ? 290.0 : bn == 192 ? 405.0 : 465.0;
    const int64_t tiles = (int64_t)((M + 255) / 256) * ((N + bn - 1) / bn);
    for (int s = 1; s <= (bn <= 128 ? 8 : 1) && s <= k_blocks; ++s) {
      Fp8Plan p;
      p.bn = bn;
      p.splits = s;
      const int cap = std::min(gemm_cluster_capacity(2 * s), sms / (2 * s));
      const double waves = std::ceil((double)tiles / cap);
      if (s > 1 && waves > 1) break;
      p.clusters = (int)std::min<int64_t>(tiles, cap);
      const int kbs = (k_blocks + s - 1) / s;
      const double power_ns = 2.0 * ((M + 255) / 256) * 256.0 * ((N + bn - 1) / bn) * bn * k_blocks * kBlockK / 2.6e6;
      p.ns = std::max({waves * kbs * kb_ns, power_ns, dram_ns}) +
             (s == 1 ? 2490.0 + 5.6 * bn : 5060.0 + 23.5 * std::max(bn - 64, 0) + 86.0 * s) + (waves - 1) * 7.8 * bn +
             (4 * s * p.clusters > sms ? (M <= 256 ? 910.0 : 450.0) : 0.0);
      if (p.ns < best.ns) best = p;
    }
  }
  return best;
}

const Fp8Plan& cached_plan(int M, int N, int K, int sms) {
  static thread_local PlanCache<Fp8Plan> cache;
  int device = 0;
  cudaGetDevice(&device);
  return cache.get(M, N, K, sms, device, make_fp8_plan);
}

template <int CHUNKS>
cudaError_t launch(const Fp8Plan& plan, const Fp8Params& p, const CUtensorMap& map_a, const CUtensorMap& map_b,
                   const CUtensorMap& map_c, cudaStream_t stream) {
  static OncePerDevice once;
  const cudaError_t opted = once([] { return opt_in(fp8_gemm_kernel<CHUNKS>, kMaxDynamicSmem, CHUNKS <= 2); });
  if (opted != cudaSuccess) return opted;
  const int total = p.m_tiles * p.n_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * plan.splits * (plan.splits > 1 ? total : plan.clusters)));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = 1024 + (size_t)p.stage_area + kTailBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)(2 * plan.splits);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, fp8_gemm_kernel<CHUNKS>, map_a, map_b, map_c, p);
}

}  // namespace

int fp8_gemm_smem(int bn, int splits) {
  const Fp8Memory m = fp8_memory(bn, splits);
  return 1024 + m.stage_area + kTailBytes;
}

Fp8GemmPlan fp8_gemm_plan(int M, int N, int K, int sms) {
  const Fp8Plan& p = cached_plan(M, N, K, sms);
  return {p.bn, p.splits};
}

cudaError_t launch_fp8_gemm(const Fp8GemmArgs& a, cudaStream_t stream) {
  if (a.M <= 0 || a.N <= 0 || a.K <= 0 || a.K % 16 != 0) return cudaErrorInvalidValue;
  const Fp8Plan& plan = cached_plan(a.M, a.N, a.K, a.sms);
  Fp8Params p = {};
  p.a_scale = a.a_scale;
  p.b_scale = a.b_scale;
  p.c = reinterpret_cast<__nv_bfloat16*>(a.c);
  p.M = a.M;
  p.N = a.N;
  p.k_blocks = (a.K + kBlockK - 1) / kBlockK;
  p.as_stride_m = a.as_stride_m;
  p.as_stride_k = a.as_stride_k;
  p.bs_stride_n = a.bs_stride_n;
  p.bs_stride_k = a.bs_stride_k;
  p.splits = plan.splits;
  p.m_tiles = (a.M + 255) / 256;
  p.n_tiles = (a.N + plan.bn - 1) / plan.bn;
  p.band = std::min(8, p.m_tiles);
  p.tma_out = (a.N % 8 == 0 && (reinterpret_cast<uintptr_t>(a.c) & 15u) == 0) ? 1 : 0;
  p.timeout_ns = a.timeout_ns;
  p.status = a.status;
  const Fp8Memory mem = fp8_memory(plan.bn, plan.splits);
  p.stages = mem.stages;
  p.stage_area = mem.stage_area;
  if (1024 + p.stage_area + kTailBytes > kMaxDynamicSmem) return cudaErrorInvalidValue;
  CUtensorMap map_a, map_b, map_c = {};
  if (!make_tensor_map(&map_a, a.a, (uint64_t)a.M, (uint64_t)a.K, 1, kRows, kBlockK, 128) ||
      !make_tensor_map(&map_b, a.b, (uint64_t)a.N, (uint64_t)a.K, 1, (uint32_t)plan.bn / 2, kBlockK, 128) ||
      (p.tma_out && !make_tensor_map(&map_c, a.c, (uint64_t)a.M, (uint64_t)a.N, 2, 32, 32, 64)))
    return cudaErrorInvalidValue;
  switch (plan.bn) {
    case 64: return launch<1>(plan, p, map_a, map_b, map_c, stream);
    case 128: return launch<2>(plan, p, map_a, map_b, map_c, stream);
    case 192: return launch<3>(plan, p, map_a, map_b, map_c, stream);
    default: return launch<4>(plan, p, map_a, map_b, map_c, stream);
  }
}

cudaError_t launch_fp8_wait_selftest(StatusWord* status, uint64_t timeout_ns, cudaStream_t stream) {
  Fp8Params p = {};
  p.timeout_ns = timeout_ns;
  p.status = status;
  fp8_wait_selftest_kernel<<<1, 32, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace b200
