// GEMM (+ bias) of one rank for sm_100a: out[M, N] = A[M, K] . W[N, K]^T, bf16 in and out, fp32 accumulation.
//
// Both kernels multiply rows of one operand (the "P side", a tensor-memory lane per row) by rows of the other (the
// "Q side", accumulator columns):
//   normal   P = A (tokens), Q = W (features): a lane holds a run of one output row
//   swapped  P = W, Q = A: for few tokens, so that the 128-row side is full and the tile is as wide as the batch
// The width `bn` of the Q side is a runtime value (a multiple of 32): the instruction descriptor, the copy boxes and
// the number of pipeline stages follow it.
//
//   gemm_tile_kernel   problems of about one wave: one CTA per tile of up to 128 P rows, or a pair (cta_group::2) per
//                      256; where there are fewer tiles than SMs, a cluster of them shares a tile, each with a part of
//                      K, and adds the parts up through distributed shared memory.
//   gemm_pair_kernel   larger ones: persistent CTA pairs (cta_group::2) on tiles of 256 P rows; the last wave, which
//                      would leave pairs idle, is dealt out by k-blocks instead of by tiles.  The largest ones run
//                      against the power limit: there a tile is 512 columns, both accumulators wide, and a quarter
//                      less operand traffic buys clock (8192 x 8192 x 28672 in a row of calls: 1280 MHz instead of the
//                      1100 with 256 columns, and 4.5 % less time).
//
// Multi-rank kernel before -> these kernels, one rank, us in a row of calls (cool, then the SM clock of a long row, held
// down at 985 W): 64 x 2880 x 360 10.2 -> 4.2 (latency: a launch and its call), 64 x 7168 x 18432 71 -> 48 (46, 1550 MHz;
// memory, 5.9 TB/s), 256 x 5120 x 12800 58 -> 40 (35, 1455 MHz; memory, then the meeting of the parts), 2048 x 2880 x 2880
// 45 -> 31 (26, 1500 MHz; 144 tiles on 74 pairs), 8192 x 8192 x 28672 3135 -> 2787 (2430, 1297 MHz).  Widths are multiples
// of 32 columns; with multiples of 64 only, 256 x 5120 x 12800 was three parts of 256 columns on 120 CTAs (40 us; two parts
// of 160 on 128 are less to exchange), 2048 x 2880 x 2880 120 tiles of 192 (33.5 us).
// Tried and level: as many pipeline stages as a part has k-blocks, which lets two launches share an SM.
//
// Warp roles of both (320 threads): 0 TMA producer, 1 MMA issuer, 2..9 epilogue, two per tensor-memory lane quarter.
// Shared memory keeps CTAs of the pair kernel, which take all of the tensor memory, alone on their SM.  Small tiles of
// the tile kernel leave room for a second CTA, so a CTA takes no more tensor memory than its accumulator: whatever fits
// on an SM by shared memory has its columns too, and no CTA ever waits for another one's.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "gemm_rs.h"
#include "per_device.h"
#include "plan_cache.h"
#include "signal.cuh"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace b200 {

namespace {

constexpr int kPRows = 128;                  // P rows per CTA
constexpr int kBK = 64;                      // 64 bf16 = one 128-byte swizzled row
constexpr int kPBytes = kPRows * kBK * 2;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kMaxStages = 12;
constexpr int kSlabBytes = 4096;             // per epilogue warp: 32 rows x 128 bytes on their way to global memory
constexpr int kTailBytes = kEpiWarps * kSlabBytes + kEpiWarps * 64 * 2 + 256;  // slabs, bias values, barriers
constexpr int kMaxDynamicSmem = 232448 - 256;  // 227 KiB less what is static
constexpr int kAccCols = 256;                // tensor-memory columns between the two accumulators
constexpr int kTmemCols = 512;               // pair kernel: both accumulators

struct LocalParams {
  const __nv_bfloat16* bias;
  float bias_scale;
  int bias_mode;      // 0 none, 1 added to the rounded product (then rounded again), 2 added in fp32
  __nv_bfloat16* out; // [M, N]
  int N;
  int P, Q;           // rows of the two operands
  int num_kb;
  int p_tiles, q_tiles, band, bn, stages;
  int rows;           // tile kernel: P rows of a CTA's tile, at most 128
  int splits;         // tile kernel: CTAs (or pairs) of a cluster that share a tile
  int part_bytes;     // tile kernel: shared memory of its own for their parts (0: they take the pipeline's)
  int tmem_cols;      // tile kernel: tensor-memory columns of its one accumulator
  int group;          // chunks of 32 columns that leave together: 2, or 1 (swapped, or `bn` is an odd number of chunks)
  int stage_area;     // tile kernel: bytes of the pipeline's stages, and of the parts where these share them
  int sk_tiles, total_tiles;  // pair kernel
  int halves;         // pair kernel: 2 = a tile is twice `bn` columns, one accumulator for each half
  float* partials;    // pair kernel: [2][pair][cta][bn / 32][8][128 rows] float4
  int64_t far_part;   // float4s between the two halves of `partials`
  uint32_t* counters; // pair kernel: [sk_tiles][cta][epilogue warp], zero between launches
  uint64_t timeout_ns;
  StatusBlock* status;
  uint64_t* trace;    // optional [gridDim.x][8]: 0 start, 1 ready, 2 tiles done, 3 exit
};

__device__ __forceinline__ void stamp(const LocalParams& p, int slot) {
  if (p.trace != nullptr) p.trace[(size_t)blockIdx.x * 8 + slot] = global_timer_ns();
}

__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort, const LocalParams& p,
                                         int detail) {
  if (ptx::mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  uint32_t spins = 0;
  while (!ptx::mbar_try_wait(bar, parity)) {
    if ((++spins & 255u) == 0) {
      if (*abort) return false;
      if (global_timer_ns() - t0 > p.timeout_ns) {
        record_status(p.status, STATUS_TIMEOUT, PHASE_GEMM_PIPELINE, -1, detail, 0, parity);
        *abort = 1;
        return false;
      }
    }
  }
  return true;
}

// The k-block runs of one pair, in the order in which every warp role goes through them: first its share of the cut
// tiles (so that their reductions hide behind the whole tiles), then its whole tiles.
struct Segments {
  int tile, kb0, kb1;
  int u, u1, next_whole;
  __device__ __forceinline__ void init(const LocalParams& p, int pair, int pairs) {
    const long long units = (long long)p.sk_tiles * p.num_kb;
    u = (int)(units * pair / pairs);
    u1 = (int)(units * (pair + 1) / pairs);
    next_whole = p.sk_tiles + pair;
  }
  __device__ __forceinline__ bool next(const LocalParams& p, int pairs) {
    if (u < u1) {
      tile = u / p.num_kb;
      kb0 = u - tile * p.num_kb;
      kb1 = min(p.num_kb, kb0 + (u1 - u));
      u += kb1 - kb0;
      return true;
    }
    tile = next_whole;
    kb0 = 0;
    kb1 = p.num_kb;
    next_whole += pairs;
    return tile < p.total_tiles;
  }
};

// Tiles are visited in bands of `band` P tiles, Q tile by Q tile, so that pairs at work at the same time share operands in L2.
__device__ __forceinline__ void tile_coords(const LocalParams& p, int tile, int& pt, int& qt) {
  const int per_band = p.band * p.q_tiles;
  const int b = tile / per_band;
  const int start = b * p.band;
  const int size = min(p.band, p.p_tiles - start);
  const int within = tile - start * p.q_tiles;
  qt = within / size;
  pt = start + within - qt * size;
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Two rounded products and their bias values, added and rounded again: the exact sum of two bf16 numbers either fits fp32
// (exponents up to 16 apart) or rounds to the larger one either way, so this is with_bias() and a rounding, in one
// instruction for both.
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t v, uint32_t b) {
  const __nv_bfloat162 s =
      __hadd2_rn(*reinterpret_cast<const __nv_bfloat162*>(&v), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&s);
}

__device__ __forceinline__ float with_bias(float v, float b, int mode) {
  if (mode == 1) return __bfloat162float(__float2bfloat16_rn(v)) + b;
  return v + b;
}

// Where an epilogue warp stands: its slab and bias values in shared memory, how many groups it has sent off, and (not
// swapped) the lane's two bias values of the group that is next.  These are asked for a group ahead, the first ones before
// the accumulator is waited for: asked for when the group's turn came, each group waited for memory once more, and narrow
// groups made that worse.  (us with a bias, then -> now; without one: 2558 x 1368 x 416 9.5 -> 8.7; 7.4, 3515 x 1048 x 744
// 12.2 -> 11.4; 10.1, 5256 x 576 x 360 9.1 -> 8.9; 7.3.  The rest is arithmetic.)
struct Emit {
  uint32_t slab, bias;
  uint32_t stores = 0;
  uint32_t two = 0;
};

__device__ __forceinline__ float bias_of_lane(const LocalParams& p, int feature) {
  if (p.bias_mode == 0 || feature >= p.N) return 0.f;
  const float b = __bfloat162float(p.bias[feature]);
  return p.bias_mode == 2 ? b * p.bias_scale : b;
}

// bias value e of packed bf16 words
__device__ __forceinline__ float bias_of_word(const LocalParams& p, const uint32_t* words, int e) {
  const float b = __uint_as_float((e & 1) ? (words[e >> 1] & 0xffff0000u) : (words[e >> 1] << 16));
  return p.bias_mode == 2 ? b * p.bias_scale : b;
}

// The lane's bias values of group g (N is a multiple of 8: both or none).
__device__ __forceinline__ uint32_t ask_bias(const LocalParams& p, int qrow, int g, int lane) {
  const int n = qrow + g * p.group * 32 + 2 * lane;
  return p.bias_mode != 0 && n < p.Q ? *reinterpret_cast<const uint32_t*>(p.bias + n) : 0u;
}

// One column group of a warp's 32 rows -- p.group chunks of 32 columns -- from fp32 to the result: bias, rounding,
// through the warp's slab, out by TMA (which clips what lies outside the result).  chunk(c, v) gives 32 columns.
template <bool SWAP, typename F>
__device__ __forceinline__ void emit_group(const LocalParams& p, const CUtensorMap* map_out, Emit& em, int g, int prow,
                                           int qrow, float lane_bias, int lane, F&& chunk) {
  const int group = SWAP ? 1 : p.group;
  const uint32_t buf = group == 1 ? em.slab + (em.stores & 1u) * (kSlabBytes / 2) : em.slab;
  ++em.stores;
  if (!SWAP && p.bias_mode != 0) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(em.bias + (uint32_t)lane * 4u), "r"(em.two) : "memory");
    em.two = ask_bias(p, qrow, g + 2, lane);
  }
  if (lane == 0) {  // the store that used this buffer has read it
    if (group == 1) ptx::bulk_wait_group_read<1>();
    else ptx::bulk_wait_group_read<0>();
  }
  __syncwarp();
#pragma unroll 1
  for (int cc = 0; cc < group; ++cc) {
    float v[32];
    chunk(g * group + cc, v);
    if (SWAP) {
      // lane = feature, v[j] = token j of the chunk.  Two lanes exchange values so that each writes the feature
      // pair of one of two tokens: rows of 64 bytes, 16 words per token, no bank conflict.
      if (p.bias_mode != 0) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = with_bias(v[j], lane_bias, p.bias_mode);
      }
      const bool odd = lane & 1;
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float mine = odd ? v[j + 1] : v[j];
        const float other = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
        const uint32_t word = odd ? pack2(other, mine) : pack2(mine, other);
        const uint32_t at = buf + (uint32_t)(j + (odd ? 1 : 0)) * 64u + (uint32_t)(lane >> 1) * 4u;
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(word) : "memory");
      }
    } else {
      uint32_t w[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) w[j] = pack2(v[2 * j], v[2 * j + 1]);
      if (p.bias_mode != 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t b[4];
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                       : "r"(em.bias + (uint32_t)(cc * 32 + j * 8) * 2u));
          if (p.bias_mode == 1) {
#pragma unroll
            for (int e = 0; e < 4; ++e) w[4 * j + e] = add_bf16x2(w[4 * j + e], b[e]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[4 * j + e] = pack2(v[8 * j + 2 * e] + bias_of_word(p, b, 2 * e),
                                   v[8 * j + 2 * e + 1] + bias_of_word(p, b, 2 * e + 1));
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // 16-byte piece cc * 4 + j of row `lane`, where the 128 (64)-byte swizzle wants it
        const uint32_t at = group == 2 ? buf + (uint32_t)lane * 128u + (uint32_t)(((cc * 4 + j) ^ (lane & 7)) << 4)
                                       : buf + (uint32_t)lane * 64u + (uint32_t)((j ^ ((lane >> 1) & 3)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(w[4 * j]), "r"(w[4 * j + 1]),
                     "r"(w[4 * j + 2]), "r"(w[4 * j + 3])
                     : "memory");
      }
    }
  }
  ptx::fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    const int x = SWAP ? prow : qrow + g * group * 32;
    const int y = SWAP ? qrow + g * 32 : prow;
    if (x < (SWAP ? p.P : p.Q) && y < (SWAP ? p.Q : p.P)) ptx::tma_store_2d(map_out, buf, x, y);
    ptx::bulk_commit_group();
  }
}

__device__ __forceinline__ void load_chunk(uint32_t taddr, float (&v)[32]) {
  uint32_t raw[32];
  ptx::tmem_ld_32x32b_x32(taddr, raw);
  ptx::tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
}

// After an abort: give copies still in flight time to land before shared memory is released.
__device__ __forceinline__ void drain_after_abort() {
  const uint64_t t0 = global_timer_ns();
  while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
}

}  // namespace

template <bool SWAP>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q,
                  const __grid_constant__ CUtensorMap map_out, const LocalParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int abort_flag;
  __shared__ uint32_t tmem_base_shared;
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform for the compiler too
  const int lane = tid & 31;
  if (tid == 0) stamp(p, 0);
  const uint32_t cta = ptx::cluster_ctarank();
  const bool leader = cta == 0;
  const int pair = (int)blockIdx.x >> 1;
  const int pairs = (int)gridDim.x >> 1;

  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_bytes = (uint32_t)p.bn * (kBK * 2 / 2);  // this CTA's part of the Q rows
  const uint32_t stage_bytes = kPBytes + (uint32_t)p.halves * q_bytes;
  const uint32_t slabs = base + (uint32_t)p.stages * stage_bytes;
  const uint32_t bias_smem = slabs + kEpiWarps * kSlabBytes;
  const uint32_t bars = bias_smem + kEpiWarps * 64 * 2;
  auto full_bar = [&](uint32_t s) { return bars + 8u * s; };
  auto empty_bar = [&](uint32_t s) { return bars + 8u * (kMaxStages + s); };
  auto tfull_bar = [&](uint32_t s) { return bars + 8u * (2 * kMaxStages + s); };
  auto tempty_bar = [&](uint32_t s) { return bars + 8u * (2 * kMaxStages + 2 + s); };

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(tfull_bar(s), 1);
      ptx::mbar_init(tempty_bar(s), 2 * kEpiWarps);
    }
    ptx::fence_mbar_init();
    ptx::fence_proxy_async_smem();
    ptx::prefetch_tensormap(&map_p);
    ptx::prefetch_tensormap(&map_q);
    ptx::prefetch_tensormap(&map_out);
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(ptx::smem_u32(&tmem_base_shared), kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();  // the other CTA's barriers exist before anything signals them
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_shared;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  if (tid == 0) stamp(p, 1);

  Segments seg;
  seg.init(p, pair, pairs);

  if (warp == 0) {
    // ---- TMA producer: this CTA's 128 P rows and half of the Q rows of every k-block -----------------
    uint32_t stage = 0, phase = 0;
    while (!abort_flag && seg.next(p, pairs)) {
      int pt, qt;
      tile_coords(p, seg.tile, pt, qt);
      const int py = pt * 256 + (int)cta * kPRows;
      const int qy = qt * p.halves * p.bn + (int)cta * (p.bn / 2);
      for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
        if (!wait_bar(empty_bar(stage), phase ^ 1u, &abort_flag, p, 100 + (int)stage)) break;
        const uint32_t sp = base + stage * stage_bytes;
        if (ptx::elect_one()) {
          if (leader) ptx::mbar_arrive_expect_tx(full_bar(stage), 2 * stage_bytes);
          ptx::tma_load_2d_pair(sp, &map_p, full_bar(stage), kb * kBK, py);
          ptx::tma_load_2d_pair(sp + kPBytes, &map_q, full_bar(stage), kb * kBK, qy);
          if (p.halves == 2) ptx::tma_load_2d_pair(sp + kPBytes + q_bytes, &map_q, full_bar(stage), kb * kBK, qy + p.bn);
        }
        __syncwarp();
        if (++stage == (uint32_t)p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: one lane of the leader drives both CTAs' tensor cores -----------------------------
    if (leader) {
      const uint32_t idesc = ptx::make_idesc_bf16_f32(256, p.bn);
      uint32_t stage = 0, phase = 0, it = 0;
      auto wait_acc = [&](uint32_t acc, uint32_t use) {
        const bool ok = wait_bar(tempty_bar(acc), (use & 1u) ^ 1u, &abort_flag, p, 200 + (int)acc);
        ptx::tcgen05_fence_after();
        return ok;
      };
      auto wait_full = [&](uint32_t s, uint32_t ph) {
        const bool ok = wait_bar(full_bar(s), ph, &abort_flag, p, 300 + (int)s);
        ptx::tcgen05_fence_after();
        return ok;
      };
      auto multiply = [&](uint32_t s, uint32_t half, uint32_t acc, bool first) {  // (one lane)
        const uint32_t sp = base + s * stage_bytes;
        const uint64_t dp = ptx::make_smem_desc_k_sw128(sp);
        const uint64_t dq = ptx::make_smem_desc_k_sw128(sp + kPBytes + half * q_bytes);
        const uint32_t d = tmem_base + acc * kAccCols;
#pragma unroll
        for (int j = 0; j < kBK / 16; ++j)  // 16 bf16 of K = 32 bytes = 2 descriptor address units
          ptx::umma_bf16_pair(d, dp + 2u * j, dq + 2u * j, idesc, (!first || j > 0) ? 1u : 0u);
      };
      auto advance = [&](uint32_t& s, uint32_t& ph) {
        if (++s == (uint32_t)p.stages) {
          s = 0;
          ph ^= 1u;
        }
      };
      for (; !abort_flag && seg.next(p, pairs); ++it) {
        bool ok = true;
        int kb = seg.kb0;
        if (p.halves == 2) {
          // As many k-blocks as the pipeline holds go into the first half's accumulator before the second half's is
          // waited for: the epilogue of the tile before is still reading that one.
          const int held = min(p.stages, p.num_kb);
          ok = wait_acc(0, it);
          uint32_t s = stage, ph = phase;
          for (int i = 0; i < held && ok; ++i) {
            ok = wait_full(s, ph);
            if (ok && ptx::elect_one()) multiply(s, 0, 0, i == 0);
            __syncwarp();
            advance(s, ph);
          }
          ok = ok && wait_acc(1, it);
          for (; kb < held && ok; ++kb) {
            if (ptx::elect_one()) {
              multiply(stage, 1, 1, kb == 0);
              ptx::umma_commit_pair(empty_bar(stage), 3);
            }
            __syncwarp();
            advance(stage, phase);
          }
          for (; kb < seg.kb1 && ok; ++kb) {
            ok = wait_full(stage, phase);
            if (ok && ptx::elect_one()) {
              multiply(stage, 0, 0, false);
              if (kb + 1 == seg.kb1) ptx::umma_commit_pair(tfull_bar(0), 3);
              multiply(stage, 1, 1, false);
              ptx::umma_commit_pair(empty_bar(stage), 3);
            }
            __syncwarp();
            advance(stage, phase);
          }
          if (!ok) break;
          if (ptx::elect_one()) {
            if (held == p.num_kb) ptx::umma_commit_pair(tfull_bar(0), 3);
            ptx::umma_commit_pair(tfull_bar(1), 3);
          }
          __syncwarp();
          continue;
        }
        const uint32_t acc = it & 1u;
        ok = wait_acc(acc, it >> 1);
        for (; kb < seg.kb1 && ok; ++kb) {
          ok = wait_full(stage, phase);
          if (ok && ptx::elect_one()) {
            multiply(stage, 0, acc, kb == seg.kb0);
            ptx::umma_commit_pair(empty_bar(stage), 3);
          }
          __syncwarp();
          advance(stage, phase);
        }
        if (!ok) break;
        if (ptx::elect_one()) ptx::umma_commit_pair(tfull_bar(acc), 3);
        __syncwarp();
      }
    }
  } else {
    // ---- epilogue ----------------------------------------------------------------------------------------
    const int ew = warp - 2;
    const int q = warp & 3;       // tensor-memory lane quarter this warp may read
    const int half = ew >> 2;
    const int chunks = p.bn / 32;
    const int group = SWAP ? 1 : p.group;  // this warp takes every second group of so many chunks
    Emit em{slabs + (uint32_t)ew * kSlabBytes, bias_smem + (uint32_t)ew * 128u};
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
    const size_t part_vecs = (size_t)chunks * 8 * kPRows;  // float4s of one CTA's half of a tile
    uint32_t it = 0;
    for (;; ++it) {
      const uint32_t acc = it & 1u;
      if (abort_flag || ((p.halves == 1 || acc == 0) && !seg.next(p, pairs))) break;
      int pt, qt;
      tile_coords(p, seg.tile, pt, qt);
      const int prow = pt * 256 + (int)cta * kPRows + q * 32;
      const int qrow = p.halves == 1 ? qt * p.bn : (2 * qt + (int)acc) * p.bn;
      const float lane_bias = SWAP ? bias_of_lane(p, prow + lane) : 0.f;
      if (!SWAP) em.two = ask_bias(p, qrow, half, lane);
      // A cut tile has two contributors: the pair that starts it, as its last piece of cut work, and the next pair,
      // as its first.  Whoever comes second, warp by warp, finds the other's accumulator in the workspace and
      // finishes the tile; nobody waits.  (A sum of two terms is the same in either order.)
      const bool cut = seg.kb1 - seg.kb0 < p.num_kb;
      const int starter = pair - (seg.kb0 > 0 ? 1 : 0);
      uint32_t* ctr = p.counters + ((size_t)(cut ? seg.tile : 0) * 2 + cta) * kEpiWarps + ew;
      float4* part = reinterpret_cast<float4*>(p.partials) + ((size_t)(cut ? starter : 0) * 2 + cta) * part_vecs + q * 32 + lane;
      int second = 0;
      if (cut) {  // as a rule the starter is second, and this is known before its accumulator is complete
        if (lane == 0) second = ld_acquire_gpu_u32(ctr) != 0;
        second = __shfl_sync(0xffffffffu, second, 0);
      }
      if (!wait_bar(tfull_bar(acc), (it >> 1) & 1u, &abort_flag, p, 400 + (int)acc)) break;
      ptx::tcgen05_fence_after();
      const uint32_t acc_addr = lane_addr + acc * kAccCols;
      auto release = [&]() {  // all reads of this accumulator are done
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(tempty_bar(acc), 0);
      };
      bool own_in_tmem = true;
      if (cut && !second) {
        // Leave the accumulator: at the far end of the starter's block if it is the next pair's, so that both can
        // be there at once.
        float4* dst = part + (seg.kb0 > 0 ? 0 : (size_t)p.far_part);
        for (int c = 0; c < chunks; ++c) {
          if (((group == 1 ? c : c / 2) & 1) != half) continue;
          float v[32];
          load_chunk(acc_addr + c * 32, v);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            __stcg(dst + (size_t)(c * 8 + j) * kPRows, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
        }
        release();
        own_in_tmem = false;
        __syncwarp();
        if (lane == 0) {
          __threadfence();
          second = atomicAdd(ctr, 1u) != 0;  // the other one came meanwhile
        }
        second = __shfl_sync(0xffffffffu, second, 0);
        if (!second) continue;
      }
      if (cut) {
        if (lane == 0) {
          __threadfence();  // what the other wrote before it counted itself in
          *ctr = 0;
        }
        __syncwarp();
      }
      const float4* theirs = part + (seg.kb0 > 0 ? (size_t)p.far_part : 0);
      const float4* mine = part + (seg.kb0 > 0 ? 0 : (size_t)p.far_part);
      float4 ahead[8];
      auto ask = [&](int c) {  // the other's share of a chunk, one chunk ahead of its use
#pragma unroll
        for (int j = 0; j < 8; ++j) ahead[j] = __ldcg(theirs + (size_t)(c * 8 + j) * kPRows);
      };
      if (cut && half * group < chunks) ask(half * group);
#pragma unroll 1
      for (int g = half; g * group < chunks; g += 2) {
        emit_group<SWAP>(p, &map_out, em, g, prow, qrow, lane_bias, lane, [&](int c, float (&v)[32]) {
          if (own_in_tmem) {
            load_chunk(acc_addr + c * 32, v);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) *reinterpret_cast<float4*>(&v[4 * j]) = __ldcg(mine + (size_t)(c * 8 + j) * kPRows);
          }
          if (cut) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              v[4 * j] += ahead[j].x;
              v[4 * j + 1] += ahead[j].y;
              v[4 * j + 2] += ahead[j].z;
              v[4 * j + 3] += ahead[j].w;
            }
            const int next = group == 2 && c == 2 * g ? c + 1 : (g + 2) * group;
            if (next < chunks) ask(next);
          }
        });
      }
      if (own_in_tmem) release();
    }
    if (lane == 0) ptx::bulk_wait_group_read<0>();
    if (tid == 64) stamp(p, 2);
  }

  if (abort_flag) drain_after_abort();
  __syncwarp();
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();  // neither CTA retires while the other may still signal its barriers or read its memory
  ptx::tcgen05_fence_after();
  if (warp == 1) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
  if (tid == 0) stamp(p, 3);
}

// One tile per CTA, up to 128 P rows by bn columns, or per CTA pair, twice the rows.  With `splits` > 1 a cluster
// shares the tile, each CTA or pair over its part of K.  When its part is complete, a CTA stores the
// columns that other members finish straight into their shared memory; after one cluster barrier every member adds
// up its columns in the order of K and writes them.  No workspace, no flags in global memory.
template <bool SWAP, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tile_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q,
                 const __grid_constant__ CUtensorMap map_out, const LocalParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int abort_flag;
  __shared__ uint32_t tmem_base_shared;
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform for the compiler too
  const int lane = tid & 31;
  if (tid == 0) stamp(p, 0);
  const int splits = p.splits;
  const int cluster_rank = PAIR || splits > 1 ? (int)ptx::cluster_ctarank() : 0;
  const int rank = PAIR ? cluster_rank >> 1 : cluster_rank;  // which part of K
  const int cta = PAIR ? cluster_rank & 1 : 0;               // which half of the pair's rows
  const int tile = (int)blockIdx.x / (PAIR ? 2 * splits : splits);
  const int kb0 = (int)((int64_t)p.num_kb * rank / splits);
  const int kb1 = (int)((int64_t)p.num_kb * (rank + 1) / splits);

  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const int q_rows = PAIR ? p.bn / 2 : p.bn;  // Q rows that this CTA brings in
  const uint32_t p_bytes = (uint32_t)p.rows * (kBK * 2);
  const uint32_t stage_bytes = p_bytes + (uint32_t)q_rows * (kBK * 2);
  const uint32_t slabs = base + (uint32_t)p.stage_area;
  const uint32_t bias_smem = slabs + kEpiWarps * kSlabBytes;
  const uint32_t bars = bias_smem + kEpiWarps * 64 * 2;
  const uint32_t parts = p.part_bytes > 0 ? bars + 256u : base;  // what the other members of the cluster send here
  auto full_bar = [&](uint32_t s) { return bars + 8u * s; };
  auto empty_bar = [&](uint32_t s) { return bars + 8u * (kMaxStages + s); };
  const uint32_t done_bar = bars + 8u * (2 * kMaxStages);

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    ptx::mbar_init(done_bar, 1);
    ptx::fence_mbar_init();
    ptx::fence_proxy_async_smem();
    ptx::prefetch_tensormap(&map_p);
    ptx::prefetch_tensormap(&map_q);
    ptx::prefetch_tensormap(&map_out);
  }
  if (warp == 1) {
    if (PAIR) {
      ptx::tmem_alloc_pair(ptx::smem_u32(&tmem_base_shared), (uint32_t)p.tmem_cols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(ptx::smem_u32(&tmem_base_shared), (uint32_t)p.tmem_cols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  if (PAIR || splits > 1) ptx::cluster_sync_all();  // every member runs before anything is stored into its memory
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = tmem_base_shared;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  if (tid == 0) stamp(p, 1);

  int pt, qt;
  tile_coords(p, tile, pt, qt);
  const int p0 = (pt * (PAIR ? 2 : 1) + cta) * p.rows;
  const int p_end = min(p.P, p0 + p.rows);
  const int q0 = qt * p.bn;

  if (warp == 0) {
    uint32_t stage = 0, phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!wait_bar(empty_bar(stage), phase ^ 1u, &abort_flag, p, 100 + (int)stage)) break;
      const uint32_t sp = base + stage * stage_bytes;
      if (ptx::elect_one()) {
        if (PAIR) {
          if (cta == 0) ptx::mbar_arrive_expect_tx(full_bar(stage), 2 * stage_bytes);
          ptx::tma_load_2d_pair(sp, &map_p, full_bar(stage), kb * kBK, p0);
          ptx::tma_load_2d_pair(sp + p_bytes, &map_q, full_bar(stage), kb * kBK, q0 + cta * q_rows);
        } else {
          ptx::mbar_arrive_expect_tx(full_bar(stage), stage_bytes);
          ptx::tma_load_2d(sp, &map_p, full_bar(stage), kb * kBK, p0);
          ptx::tma_load_2d(sp + p_bytes, &map_q, full_bar(stage), kb * kBK, q0);
        }
      }
      __syncwarp();
      if (++stage == (uint32_t)p.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (cta == 0) {
      const uint32_t idesc = ptx::make_idesc_bf16_f32(PAIR ? 256 : kPRows, p.bn);
      const uint16_t both = (uint16_t)(3u << (2 * rank));  // the pair's CTAs in the cluster
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = wait_bar(full_bar(stage), phase, &abort_flag, p, 300 + (int)stage);
        if (!ok) break;
        ptx::tcgen05_fence_after();
        const uint32_t sp = base + stage * stage_bytes;
        // (a tile of fewer than 128 rows is followed by other data: it gives rows of the accumulator nobody reads)
        const uint64_t dq = ptx::make_smem_desc_k_sw128(sp + p_bytes);
        const uint64_t dp = ptx::make_smem_desc_k_sw128(sp);
        if (ptx::elect_one()) {
#pragma unroll
          for (int j = 0; j < kBK / 16; ++j) {  // 16 bf16 of K = 32 bytes = 2 descriptor address units
            const uint32_t more = (kb > kb0 || j > 0) ? 1u : 0u;
            if (PAIR) ptx::umma_bf16_pair(tmem_base, dp + 2u * j, dq + 2u * j, idesc, more);
            else ptx::umma_bf16(tmem_base, dp + 2u * j, dq + 2u * j, idesc, more);
          }
          if (PAIR) ptx::umma_commit_pair(empty_bar(stage), both);
          else ptx::umma_commit(empty_bar(stage));
        }
        __syncwarp();
        if (++stage == (uint32_t)p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok && ptx::elect_one()) {
        if (PAIR) ptx::umma_commit_pair(done_bar, both);
        else ptx::umma_commit(done_bar);
      }
    }
    __syncwarp();
  }

  const int ew = warp - 2;
  const int q = warp & 3;
  const int half = ew >> 2;
  const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
  bool alive = true;
  if (warp >= 2) {
    const int prow = p0 + q * 32;
    const float lane_bias = SWAP ? bias_of_lane(p, prow + lane) : 0.f;
    Emit em{slabs + (uint32_t)ew * kSlabBytes, bias_smem + (uint32_t)ew * 128u};
    if (!SWAP && splits == 1) em.two = ask_bias(p, q0, half, lane);
    alive = wait_bar(done_bar, 0, &abort_flag, p, 400);
    ptx::tcgen05_fence_after();
    if (splits == 1 && alive && q * 32 < p.rows) {  // not split: whole groups of 32 rows
      for (int g = half; g * (SWAP ? 1 : p.group) < p.bn / 32; g += 2)
        emit_group<SWAP>(p, &map_out, em, g, prow, q0, lane_bias, lane,
                         [&](int c, float (&v)[32]) { load_chunk(lane_addr + c * 32, v); });
      if (lane == 0) ptx::bulk_wait_group_read<0>();
    }
  }

  if (splits > 1) {
    // columns [r * per, (r + 1) * per) are finished by member r; its memory holds [member][per / 4][128 rows] float4
    const int per = ((p.bn / 8 + splits - 1) / splits) * 8;
    if (p.part_bytes == 0) ptx::cluster_sync_all();  // every member is done with the stages that the parts go into
    if (warp >= 2 && alive && q * 32 < p.rows) {
      for (int c = half; c < p.bn / 32; c += 2) {
        float v[32];
        load_chunk(lane_addr + c * 32, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int col = c * 32 + j * 8;
          const int owner = col / per;
          const uint32_t to = (uint32_t)(PAIR ? 2 * owner + cta : owner);
          const uint32_t at = parts + (uint32_t)((rank * (per / 4) + (col - owner * per) / 4) * kPRows + q * 32 + lane) * 16u;
          ptx::st_cluster_v4(at, to, v[8 * j], v[8 * j + 1], v[8 * j + 2], v[8 * j + 3]);
          ptx::st_cluster_v4(at + kPRows * 16u, to, v[8 * j + 4], v[8 * j + 5], v[8 * j + 6], v[8 * j + 7]);
        }
      }
    }
    __syncwarp();
    ptx::cluster_sync_all();
    if (warp >= 2 && alive && q * 32 < p.rows) {
      const int c_lo = rank * per;
      const int c_hi = min(p.bn, c_lo + per);
      const int prow = p0 + q * 32 + lane;
      const float lane_bias = SWAP ? bias_of_lane(p, prow) : 0.f;
      for (int col = c_lo + half * 8; col < c_hi; col += 16) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = 0.f;
        const uint32_t at = parts + (uint32_t)(((col - c_lo) / 4) * kPRows + q * 32 + lane) * 16u;
        for (int m = 0; m < splits; ++m) {  // ascending k
          const uint32_t from = at + (uint32_t)m * (uint32_t)(per / 4) * kPRows * 16u;
          float f[8];
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3])
                       : "r"(from));
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7])
                       : "r"(from + kPRows * 16u));
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] += f[e];
        }
        if (prow >= p_end) continue;
        const int qc = q0 + col;
        if (SWAP) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (qc + e >= p.Q) break;
            const float f = p.bias_mode ? with_bias(v[e], lane_bias, p.bias_mode) : v[e];
            p.out[(size_t)(qc + e) * p.N + prow] = __float2bfloat16_rn(f);
          }
        } else if (qc < p.Q) {  // N is a multiple of 8: all eight or none
          if (p.bias_mode != 0) {
            const uint4 raw = *reinterpret_cast<const uint4*>(p.bias + qc);
            const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = with_bias(v[e], bias_of_word(p, words, e), p.bias_mode);
          }
          *reinterpret_cast<uint4*>(p.out + (size_t)prow * p.N + qc) =
              make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
        }
      }
    }
  }
  if (tid == 64) stamp(p, 2);

  if (abort_flag) drain_after_abort();
  __syncwarp();
  ptx::tcgen05_fence_before();
  __syncthreads();
  // neither CTA of a pair retires while the other may still signal its barriers or read its memory
  if (PAIR && splits == 1) ptx::cluster_sync_all();
  ptx::tcgen05_fence_after();
  if (warp == 1) {
    if (PAIR) ptx::tmem_dealloc_pair(tmem_base, (uint32_t)p.tmem_cols);
    else ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
  if (tid == 0) stamp(p, 3);
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
constexpr int kMaxSplits = 16;

namespace {
struct ClusterCapacities {
  int n[kMaxSplits + 1] = {0};  // by size; 0: not asked for yet
};
ClusterCapacities& cluster_capacities() {  // of the current device
  static thread_local ClusterCapacities cache[16];
  int dev = 0;
  cudaGetDevice(&dev);
  return cache[dev & 15];
}
int cluster_capacity(ClusterCapacities& known, int size) {
  int& n = known.n[size];
  if (n > 0) return n;
  auto kernel = gemm_tile_kernel<true, false>;
  opt_in(kernel, kMaxDynamicSmem, true);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(size * 16));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kMaxDynamicSmem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = size <= 8 ? std::max(1, 100 / size) : 1;
  }
  return n;
}
}  // namespace

int gemm_cluster_capacity(int size) { return cluster_capacity(cluster_capacities(), size); }

namespace {

struct Plan {
  bool persistent = false, swap = false;
  bool pair = false;                  // tile kernel: a CTA pair per tile
  int rows = 128, bn = 256, splits = 1;
  int pairs = 1, sk_tiles = 0, halves = 1;  // pair kernel
  int p_tiles = 0, q_tiles = 0;
  double ns = 1e300;
};

// How a CTA of the tile kernel divides its shared memory, and the tensor memory it takes.
struct TileMemory {
  int stages, part_bytes, stage_area, smem, tmem_cols;  // (see LocalParams)
};
TileMemory tile_memory(int rows, int bn, int splits, bool pair) {
  TileMemory t;
  const int stage_bytes = (rows + (pair ? bn / 2 : bn)) * kBK * 2;
  const int room = kMaxDynamicSmem - 1024 - kTailBytes;
  const int parts = splits > 1 ? splits * ((bn / 8 + splits - 1) / splits) * 8 * kPRows * 4 : 0;
  // the parts of a split tile in memory of their own, unless too little would be left for the pipeline
  t.part_bytes = (room - parts) / stage_bytes >= 5 ? parts : 0;
  t.stages = std::min(kMaxStages, (room - t.part_bytes) / stage_bytes);
  t.stage_area = t.stages * stage_bytes;  // (a multiple of 1024, as the slabs behind it need)
  if (t.part_bytes == 0) t.stage_area = std::max(t.stage_area, parts);
  t.smem = 1024 + t.stage_area + kTailBytes + t.part_bytes;
  t.tmem_cols = 32;  // an allocation is a power of two, at least 32
  while (t.tmem_cols < bn) t.tmem_cols *= 2;
  return t;
}

int pair_stage_bytes(int bn, int halves) { return kPBytes + halves * bn * kBK; }
int pair_stages(int bn, int halves) {
  return std::min(kMaxStages, (kMaxDynamicSmem - 1024 - kTailBytes) / pair_stage_bytes(bn, halves));
}
int pair_smem(int bn, int halves) { return 1024 + pair_stages(bn, halves) * pair_stage_bytes(bn, halves) + kTailBytes; }

int ctas_of(const Plan& p) { return p.splits * (p.pair ? 2 : 1); }  // CTAs that share a tile
int grid_ctas(const Plan& p) { return p.persistent ? 2 * p.pairs : p.p_tiles * p.q_tiles * ctas_of(p); }

// Time model in ns.  What it charges persistent pairs, measured on a B200:
//   a 128-byte row of a k-block takes an SM 1 ns to bring in, 1.6 when the rows of the matrix do not start on cache lines;
//   128 x 256 x 64 takes a tensor core 280 ns, all tensor cores together do 1.45 PFLOP/s in a row of calls (the power
//   limit; 1.55 where a launch comes alone); a k-block costs its issuing warp 150 ns; 6.6 TB/s of HBM; then what a launch
//   costs before and after its k-blocks.
// The tile kernel's terms are fitted (below).
// A size that is new to the thread pays for the search: 1.5 to 2.6 us, because a candidate whose lower bound is above the
// best so far is not worked out, and the current device is asked for once (10 to 13 us without the two; the same plans).
Plan make_local_plan(int M, int N, int K, int sms) {
  const int num_kb = (K + kBK - 1) / kBK;
  const double operand_bytes = 2.0 * ((double)M * K + (double)N * K);
  const double dram_ns = (operand_bytes + 2.0 * M * N) / 6600.0;
  const double row_ns = K % kBK == 0 ? 1.0 : 1.6;
  // ... and the narrower the tile, the more of the power goes into moving operands: `rows_per_col` is what a CTA brings
  // in per k-block, relative to a pair's 256 rows for 256 columns
  auto power_ns = [&](double rows, double cols, double rows_per_col, double pflops) {
    return 2.0 * rows * cols * num_kb * kBK / (pflops * 1e6) * (1.0 + 0.26 * (rows_per_col - 1.0));
  };
  Plan best;
  ClusterCapacities& capacities = cluster_capacities();
  auto keep = [&](const Plan& p) {
    if (p.ns < best.ns) best = p;
  };
  auto consider_tile = [&](bool swap, bool pair, int bn) {
    Plan p;
    p.swap = swap;
    p.pair = pair;
    p.bn = bn;
    const int P = swap ? N : M;
    const int halves = pair ? 2 : 1;  // tile height in units of `rows`
    p.q_tiles = ((swap ? M : N) + bn - 1) / bn;
    const int q_rows = bn / halves;
    for (int s = 1; s <= std::min(kMaxSplits / halves, num_kb); ++s) {
      const double ends_ns =
          (s == 1 ? 2580.0 + 6.6 * bn : 3980.0 + 30.0 * std::max(bn - 64, 0) + 70.0 * s) + (pair ? 220.0 : 0.0);
      if (s > 1 && dram_ns * 0.825 + ends_ns >= best.ns) break;  // (and no larger s does better)
      p.splits = s;
      const int cap = ctas_of(p) == 1 ? sms : cluster_capacity(capacities, ctas_of(p));
      // Lower tiles when that many clusters fit at once and full ones would leave SMs without work: a share of the
      // weight for everybody.  (Not split, tiles end on the 32 rows of an epilogue warp.)
      p.rows = 128;
      if (swap) {
        const int step = s == 1 ? 32 : 8;
        const int fit = halves * std::max(cap / p.q_tiles, 1);
        p.rows = std::min(128, ((P + fit - 1) / fit + step - 1) / step * step);
      }
      p.p_tiles = (P + halves * p.rows - 1) / (halves * p.rows);
      const int64_t tiles = (int64_t)p.p_tiles * p.q_tiles;
      if (tiles > 4 * (int64_t)cap) continue;
      const int waves = ((int)tiles + cap - 1) / cap;
      const int kbs = (num_kb + s - 1) / s;
      const int stages = std::min(kMaxStages, (kMaxDynamicSmem - 1024 - kTailBytes) / ((p.rows + q_rows) * kBK * 2));
      // Fitted to 2179 timed plans of 190 drawn sizes (the plan it picks is 3 % from the best of each size).  What limits
      // a tile's main loop does not add up, but does not hide behind one another either: a copy that waits for memory
      // also waits for its turn in the SM.
      const double kb_ns =
          std::max({(K % kBK == 0 ? 0.55 : 1.15) * (p.rows + q_rows), 246.0 * bn / 256.0, 140.0, 1200.0 / stages});
      const double limits[3] = {waves * kbs * kb_ns, dram_ns * 0.825,
                                power_ns(p.p_tiles * halves * 128.0, (double)p.q_tiles * bn, (128.0 + q_rows) / bn, 1.55)};
      const double largest = std::max({limits[0], limits[1], limits[2]});
      if (largest + ends_ns + (waves - 1) * 4000.0 >= best.ns) continue;  // (it is more than that)
      double cubes = 0.0;
      for (double t : limits) cubes += t * t * t;
      p.ns = std::cbrt(cubes) + ends_ns + (waves - 1) * 4000.0;
      keep(p);
    }
  };
  auto consider_pair = [&](bool swap, int bn, int halves) {
    Plan p;
    p.persistent = true;
    p.swap = swap;
    p.bn = bn;
    p.p_tiles = ((swap ? N : M) + 255) / 256;
    p.halves = halves;
    const int cols = halves * bn;
    p.q_tiles = ((swap ? M : N) + cols - 1) / cols;
    const int64_t tiles = (int64_t)p.p_tiles * p.q_tiles;
    p.pairs = (int)std::min<int64_t>(tiles, std::min(sms / 2, kGemmLocalMaxPairs));
    if (halves == 1 && tiles == p.pairs) return;  // one wave: the tile kernel's pairs do the same 8 % faster
    // A wave takes as long as one of its tiles, or as the power for all of them: a last wave of few tiles has power to
    // spare, and its tiles still take their time (2048 x 5120 x 12800: 231 us in 2.2 waves of 256 columns, 214 in 2.9 of
    // 192).
    const double wave_ns = power_ns(256.0 * p.pairs, cols, (128.0 + cols / 2) / cols, 1.45);
    const double tile_ns = num_kb * std::max({row_ns * (128 + cols / 2), 280.0 * cols / 256.0, 150.0});
    const int64_t whole = tiles / p.pairs, last = tiles % p.pairs;
    const int64_t waves = whole + (last > 0 ? 1 : 0);
    p.sk_tiles = 0;
    const double last_ns = last > 0 ? std::max(tile_ns, wave_ns * last / p.pairs) : 0.0;
    p.ns = std::max(whole * std::max(tile_ns, wave_ns) + last_ns, dram_ns) + 3400.0 + 9.0 * cols;
    // With both accumulators in one tile, 5.5 us of its epilogue do not run beside products (all pairs store at once).
    if (halves == 2) p.ns += waves * 5500.0;
    keep(p);
    if (halves == 1 && whole > 0 && last != 0) {
      p.sk_tiles = (int)last + p.pairs;
      // The parts of the cut tiles go through memory: 5 us in all, and time by how many pairs' work is cut up.  (With 2.5 us
      // 2348 x 2144 x 1504 was cut and took 21.4 us where whole tiles of 192 columns take 16.5; of 240 drawn sizes, the 24
      // that are still cut gain 7 % on whole tiles.)  Pairs at work on different parts of K share no operands: what L2 does
      // not hold comes from memory for every tile (1923 x 5056 x 19824: 429 us cut, 335 in whole tiles of 192 columns).
      const double cut = (double)last / p.pairs;
      const double apart_ns = operand_bytes > 126e6 ? 0.4 * p.sk_tiles * num_kb * (256.0 + cols) * kBK * 2 / 6600.0 : 0.0;
      const double tiles_ns = (double)tiles / p.pairs * std::max(tile_ns, wave_ns) * (1.05 + 0.3 * cut);
      p.ns = std::max(tiles_ns, dram_ns) + apart_ns + 3400.0 + 9.0 * bn + 5000.0;
      keep(p);
    }
  };
  for (int bn = 64; bn <= 256; bn += 32) {
    for (bool pair : {false, true}) consider_tile(false, pair, bn);
    consider_pair(false, bn, 1);
  }
  consider_pair(false, 256, 2);
  const int fewest = (M + 255) / 256;
  for (int parts = fewest; parts <= std::min(fewest + 3, (M + 31) / 32); ++parts) {
    const int bn = ((M + parts - 1) / parts + 31) / 32 * 32;
    for (bool pair : {false, true}) consider_tile(true, pair, bn);
    consider_pair(true, bn, 1);
  }
  consider_pair(true, 256, 2);
  return best;
}

const Plan& cached_plan(int M, int N, int K, int sms, int device) {
  static thread_local PlanCache<Plan> cache;
  return cache.get(M, N, K, sms, device, make_local_plan);
}
const Plan& cached_plan(int M, int N, int K, int sms) {
  int device = 0;
  cudaGetDevice(&device);
  return cached_plan(M, N, K, sms, device);
}

bool common_params(LocalParams& p, const GemmLocalArgs& a, const Plan& plan, int p_rows, int q_rows, CUtensorMap* map_p,
                   CUtensorMap* map_q, CUtensorMap* map_out) {
  const bool swap = plan.swap;
  p = LocalParams{};
  p.bias = reinterpret_cast<const __nv_bfloat16*>(a.bias);
  p.bias_scale = a.bias_scale;
  p.bias_mode = a.bias == nullptr ? 0 : (a.bias_at_source ? 1 : 2);
  p.out = reinterpret_cast<__nv_bfloat16*>(a.out);
  p.N = a.N;
  p.P = swap ? a.N : a.M;
  p.Q = swap ? a.M : a.N;
  p.num_kb = (a.K + kBK - 1) / kBK;
  p.p_tiles = plan.p_tiles;
  p.q_tiles = plan.q_tiles;
  p.band = std::min(8, plan.p_tiles);
  p.bn = plan.bn;
  p.group = swap || plan.bn % 64 != 0 ? 1 : 2;
  p.rows = plan.rows;
  p.splits = plan.splits;
  p.timeout_ns = a.timeout_ns;
  p.status = a.status;
  // A grid of several waves may have more CTAs than the trace has rows: no stamps then.  (Asked here, because the same
  // question in the kernel made every launch of the tile kernel 0.05 to 0.1 us longer.)
  p.trace = grid_ctas(plan) <= a.trace_ctas ? a.trace : nullptr;
  return make_tensor_map(map_p, swap ? a.w : a.a, (uint64_t)p.P, (uint64_t)a.K, 2, (uint32_t)p_rows, kBK, 128) &&
         make_tensor_map(map_q, swap ? a.a : a.w, (uint64_t)p.Q, (uint64_t)a.K, 2, (uint32_t)q_rows, kBK, 128) &&
         make_tensor_map(map_out, a.out, (uint64_t)a.M, (uint64_t)a.N, 2, 32, (uint32_t)p.group * 32, swap ? 0 : p.group * 64);
}

template <typename K>
cudaError_t launch(K kernel, const LocalParams& p, int ctas, int cluster, size_t smem, cudaStream_t stream,
                   const CUtensorMap& map_p, const CUtensorMap& map_q, const CUtensorMap& map_out) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, map_p, map_q, map_out, p);
}

template <bool SWAP>
cudaError_t launch_pair(const GemmLocalArgs& a, const Plan& plan, cudaStream_t stream) {
  LocalParams p;
  CUtensorMap map_p, map_q, map_out;
  if (!common_params(p, a, plan, kPRows, plan.bn / 2, &map_p, &map_q, &map_out)) return cudaErrorInvalidValue;
  p.halves = plan.halves;
  if (plan.halves == 2) p.band = std::min(12, plan.p_tiles);  // 12 x 6 tiles of 256 x 512: as square as 74 pairs come
  p.stages = pair_stages(plan.bn, plan.halves);
  p.sk_tiles = plan.sk_tiles;
  p.total_tiles = plan.p_tiles * plan.q_tiles;
  p.partials = a.partials;
  p.far_part = (int64_t)(kGemmLocalPartialBytes / 2 / 16);
  p.counters = a.counters;
  static OncePerDevice once;
  const cudaError_t opted = once([] { return opt_in(gemm_pair_kernel<SWAP>, kMaxDynamicSmem, false); });
  if (opted != cudaSuccess) return opted;
  const size_t smem = (size_t)pair_smem(plan.bn, plan.halves);
  return launch(gemm_pair_kernel<SWAP>, p, grid_ctas(plan), 2, smem, stream, map_p, map_q, map_out);
}

template <bool SWAP, bool PAIR>
cudaError_t launch_tile(const GemmLocalArgs& a, const Plan& plan, cudaStream_t stream) {
  LocalParams p;
  CUtensorMap map_p, map_q, map_out;
  const int q_rows = PAIR ? plan.bn / 2 : plan.bn;
  if (!common_params(p, a, plan, plan.rows, q_rows, &map_p, &map_q, &map_out)) return cudaErrorInvalidValue;
  const TileMemory mem = tile_memory(plan.rows, plan.bn, plan.splits, PAIR);
  p.part_bytes = mem.part_bytes;
  p.stages = mem.stages;
  p.stage_area = mem.stage_area;
  p.tmem_cols = mem.tmem_cols;
  if (p.stages < 2 || mem.smem > kMaxDynamicSmem) return cudaErrorInvalidValue;
  static OncePerDevice once;
  const cudaError_t opted = once([] { return opt_in(gemm_tile_kernel<SWAP, PAIR>, kMaxDynamicSmem, true); });
  if (opted != cudaSuccess) return opted;
  return launch(gemm_tile_kernel<SWAP, PAIR>, p, grid_ctas(plan), ctas_of(plan), (size_t)mem.smem, stream, map_p, map_q,
                map_out);
}

}  // namespace

SmShare gemm_tile_share(int rows, int bn, int splits, bool pair) {
  const TileMemory t = tile_memory(rows, bn, splits, pair);
  return {t.smem, t.tmem_cols};
}
SmShare gemm_pair_share(int bn, int halves) { return {pair_smem(bn, halves), kTmemCols}; }

GemmLocalPlan gemm_local_plan(int M, int N, int K, int sms) {
  const Plan& p = cached_plan(M, N, K, sms);
  const bool own_parts = !p.persistent && tile_memory(p.rows, p.bn, p.splits, p.pair).part_bytes > 0;
  return {p.persistent, p.swap, p.persistent || p.pair, own_parts, p.rows, p.bn, p.splits, p.halves, p.sk_tiles,
          grid_ctas(p)};
}

cudaError_t launch_gemm_local(GemmLocalArgs& a, int device, const std::function<void(GemmLocalArgs&)>& workspace,
                              cudaStream_t stream) {
  if (a.M <= 0 || a.N <= 0 || a.K <= 0 || a.K % 8 != 0 || a.N % 8 != 0) return cudaErrorInvalidValue;
  Plan plan = cached_plan(a.M, a.N, a.K, a.sms, device);
  if (plan.persistent) {
    if (plan.sk_tiles > 0) workspace(a);
    if (a.partials == nullptr) plan.sk_tiles = 0;
    return plan.swap ? launch_pair<true>(a, plan, stream) : launch_pair<false>(a, plan, stream);
  }
  if (plan.pair) return plan.swap ? launch_tile<true, true>(a, plan, stream) : launch_tile<false, true>(a, plan, stream);
  return plan.swap ? launch_tile<true, false>(a, plan, stream) : launch_tile<false, false>(a, plan, stream);
}

}  // namespace b200
