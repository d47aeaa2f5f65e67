// MoE dispatch and combine when one rank holds every expert.
//
// With a single rank no row crosses a link, so nothing of the multi-rank protocol is needed: no
// landing buffer, no records for an owner to read back, no flags, no grid barrier.  One ordinary
// launch turns expert ids into slots and writes the rows to their final place; combine gathers them
// by the route table.  The layouts are those of the multi-rank kernels (rows of an expert in
// (token, k) order; 5-int metadata; per-expert counts).
//
// Both kernels may start before the previous kernel of the stream has ended (programmatic dependent launch): nothing
// is read or written before grid_dep_wait(), which makes that kernel's stores visible.  Ids, routes, weights and whole
// vectors are read past L1 (ld.global.cg), as nothing comes back for them; ragged rows, element by element, are not.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "moe.h"
#include "moe_common.cuh"
#include "signal.cuh"
#include "sm100_ptx.cuh"

namespace b200 {

namespace {

using namespace moe;

constexpr int kMetaDim = 5;
constexpr int kPieceVecs = 64;  // a warp's share of a row: 1 KiB, two 16-byte vectors per lane
__device__ __forceinline__ void stamp_cta0(uint64_t* trace, int slot) {
  if (trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0) trace[slot] = global_timer_ns();
}
__device__ __forceinline__ void stamp_last(uint64_t* trace) {
  if (trace != nullptr && threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned long long*>(trace + 7), global_timer_ns());
}

// acc[0..1] += y[0..1] * w, as one packed instruction (two fp32 FMAs, each rounded as fmaf rounds).
__device__ __forceinline__ void fma2(float2& acc, const float2& y, float w) {
  const float2 ww = make_float2(w, w);
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(acc))
      : "l"(reinterpret_cast<const unsigned long long&>(y)), "l"(reinterpret_cast<const unsigned long long&>(ww)));
}

// The expert's output for 16 bytes of a row: x * scale, rounded to T as if it had been stored.
template <typename T>
__device__ __forceinline__ void expert_output(const int4& raw, float scale, float2* y) {
  constexpr int N = Vec16<T>::N;
  float f[N];
#pragma unroll
  for (int e = 0; e < N; ++e) f[e] = 0.f;
  fma_vec<T>(f, scale_vec<T>(raw, scale), 1.f);
#pragma unroll
  for (int e = 0; e < N / 2; ++e) y[e] = make_float2(f[2 * e], f[2 * e + 1]);
}

template <typename T>
__device__ __forceinline__ int4 pack_pairs(const float2* acc) {
  return pack_vec<T>(reinterpret_cast<const float*>(acc));
}

// What a CTA of the dispatch kernel owns.
struct Share {
  int lo, hi;   // items
  int t0;       // first token
  int32_t* rows;  // shared memory: final row of every entry of tokens t0, t0 + 1, ..., or -1
};

// First half of the dispatch kernel: the CTA's share, the final rows of its entries (in shared memory), and
// the route table, metadata and counts in global memory.  Called by all threads; ends with the rows visible.
//
// Work is T x P items (token, piece of its row); CTA b owns the items [b I / G, (b + 1) I / G) and so the
// tokens they touch.  It counts the entries of all EARLIER tokens per expert by reading their ids itself (at
// most 128 KiB, out of L2) instead of meeting the other CTAs on a barrier, and ranks its own entries with one
// warp.  Neighbouring CTAs may share a token; its metadata belongs to the CTA with its first piece.
template <int THREADS>
__device__ __forceinline__ void assign_rows(const MoeLocalDispatchParams& p, int32_t* smem, Share& sh) {
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int E = p.num_experts;
  const int k = p.k;
  const int P = p.pieces;
  const int copies = p.hist_copies;
  int32_t* s_hist = smem;  // [copies][E]; after the count, row 0 holds the sums
  int32_t* s_ids = smem + copies * E;
  int32_t* s_rows = s_ids + p.cap;
  const int t1 = (sh.hi + P - 1) / P;
  const int i0 = sh.t0 * k;
  const int m = sh.hi > sh.lo ? t1 * k - i0 : 0;  // own entries
  sh.rows = s_rows;

  for (int e = tid; e < copies * E; e += THREADS) s_hist[e] = 0;
  for (int j = tid; j < m; j += THREADS) {
    int e = __ldcg(p.indices + i0 + j);
    if (e < 0 || e >= E) {
      record_status(p.status, STATUS_BAD_INDEX, PHASE_NONE, -1, i0 + j, p.epoch, (uint64_t)(int64_t)e);
      e = -1;
    }
    s_ids[j] = e;
  }
  __syncthreads();
  {
    // skewed routing has many lanes of a warp add to the same expert: spread them over the copies
    int32_t* hist = s_hist + (lane & (copies - 1)) * E;
    auto count = [&](int e) {
      if (e >= 0 && e < E) atomicAdd(&hist[e], 1);
    };
    int done = 0;
    if ((reinterpret_cast<uintptr_t>(p.indices) & 15u) == 0) {
      const int4* ids4 = reinterpret_cast<const int4*>(p.indices);
      const int n4 = i0 >> 2;
      constexpr int kFly = 8;  // loads in flight per thread
      for (int q0 = tid; q0 < n4; q0 += THREADS * kFly) {
        int4 a[kFly];
#pragma unroll
        for (int u = 0; u < kFly; ++u) {
          const int q = q0 + u * THREADS;
          a[u] = q < n4 ? __ldcg(ids4 + q) : make_int4(-1, -1, -1, -1);
        }
#pragma unroll
        for (int u = 0; u < kFly; ++u) {
          count(a[u].x);
          count(a[u].y);
          count(a[u].z);
          count(a[u].w);
        }
      }
      done = n4 << 2;
    }
    for (int i = done + tid; i < i0; i += THREADS) count(__ldcg(p.indices + i));
  }
  __syncthreads();
  if (copies > 1) {
    for (int e = tid; e < E; e += THREADS) {
      int sum = s_hist[e];
      for (int c = 1; c < copies; ++c) sum += s_hist[c * E + e];
      s_hist[e] = sum;
    }
    __syncthreads();
  }
  stamp_cta0(p.trace_d, 1);
  if (tid < 32) {
    for (int base = 0; base < m; base += 32) {
      const int j = base + lane;
      const int e = j < m ? s_ids[j] : -1;
      const unsigned active = __ballot_sync(0xffffffffu, e >= 0);
      int slot = -1;
      if (e >= 0) {
        const unsigned same = __match_any_sync(active, e);
        const int before = __popc(same & ((1u << lane) - 1u));
        const int cur = s_hist[e];
        __syncwarp(active);
        slot = cur + before;
        if (before == 0) s_hist[e] = cur + __popc(same);
      }
      __syncwarp();
      int row = -1;
      if (e >= 0) {
        if (slot < p.max_recv) row = e * p.max_recv + slot;
        else record_status(p.status, STATUS_BAD_INDEX, PHASE_NONE, 0, i0 + j, p.epoch, (uint64_t)slot);
      }
      if (j < m) s_rows[j] = row;
    }
  }
  __syncthreads();
  stamp_cta0(p.trace_d, 2);

  // route table, metadata rows (global expert, source rank, token, k, 0) and counts
  const int j_lo = ((sh.lo + P - 1) / P) * k - i0;  // entries of tokens whose first piece is this CTA's
  for (int j = max(j_lo, 0) + tid; j < m; j += THREADS) {
    const int row = s_rows[j];
    const int i = i0 + j;
    p.route[i] = make_int2(row >= 0 ? 0 : -1, row);
    if (row >= 0) {
      int32_t* meta = p.expert_meta + (size_t)row * kMetaDim;
      meta[0] = s_ids[j];
      meta[1] = 0;
      meta[2] = i / k;
      meta[3] = i % k;
      meta[4] = 0;
    }
  }
  if (blockIdx.x == gridDim.x - 1)
    for (int e = tid; e < E; e += THREADS) p.expert_num_tokens[e] = min(s_hist[e], p.max_recv);
  stamp_cta0(p.trace_d, 3);
  stamp_cta0(p.trace_d, 4);
  stamp_cta0(p.trace_d, 5);
}

__device__ __forceinline__ Share share_of_cta(const MoeLocalDispatchParams& p) {
  Share sh;
  const long long items = (long long)p.num_tokens * p.pieces;
  sh.lo = (int)(items * blockIdx.x / gridDim.x);
  sh.hi = (int)(items * (blockIdx.x + 1) / gridDim.x);
  sh.t0 = sh.lo / p.pieces;
  sh.rows = nullptr;
  return sh;
}

__device__ __forceinline__ void final_stamps(const MoeLocalDispatchParams& p, bool fused) {
  stamp_cta0(p.trace_d, 6);
  stamp_last(p.trace_d);
  if (fused) {
    stamp_cta0(p.trace_c, 2);
    stamp_cta0(p.trace_c, 3);
    stamp_last(p.trace_c);
  }
}

}  // namespace

// FUSED: the caller wants dispatch -> y = x * scale -> combine.  The expert op is
// elementwise, so its result and the weighted sum over the token's k entries are formed from the values that
// have just been stored to the expert rows; they are not written out and read back.
//
// Every warp takes one 1 KiB piece at a time through registers; the first is on its way while the slots are
// worked out, the next is asked for before the stores of the current one.  Large problems are bound by the row
// stores: 268 MB (4096 tokens, top-6, hidden 4096) in 55 us, where a bare copy of the same pattern takes 48 to
// 51.  Moving the pieces through shared memory with bulk copies measured 53 us there but 67 us (against 59)
// for dispatch + combine of 2047 tokens.  Small ones are bound by the chain ids -> counts -> slots -> stores.
template <typename T, bool FUSED, int THREADS>
__global__ void __launch_bounds__(THREADS) moe_local_dispatch_kernel(const MoeLocalDispatchParams p) {
  constexpr int kThreads = THREADS, kWarps = kThreads / 32;
  constexpr int kLaneVecs = kPieceVecs / 32;
  static_assert(kLaneVecs == 2, "the copy loop is written for two vectors per lane");
  extern __shared__ __align__(128) uint8_t smem_local[];
  const int lane = threadIdx.x & 31;
  const int k = p.k;
  const int P = p.pieces;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  stamp_cta0(p.trace_d, 0);
  Share sh = share_of_cta(p);
  const int nv = (int)(p.row_bytes >> 4);
  int item = sh.lo + (int)(threadIdx.x >> 5);
  int4 next[kLaneVecs];
  auto load_piece = [&](int item) {
    const int t = item / P;
    const int v0 = (item - t * P) * p.piece_vecs;
    const int v1 = min(nv, v0 + p.piece_vecs);
    const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(p.x) + (size_t)t * p.row_bytes);
#pragma unroll
    for (int u = 0; u < kLaneVecs; ++u)
      if (v0 + lane + 32 * u < v1) next[u] = __ldcg(src + v0 + lane + 32 * u);
  };
  if (p.vec && item < sh.hi) load_piece(item);

  assign_rows<kThreads>(p, reinterpret_cast<int32_t*>(smem_local), sh);
  if (FUSED) {
    stamp_cta0(p.trace_c, 0);
    stamp_cta0(p.trace_c, 1);
  }
  uint8_t* ex = reinterpret_cast<uint8_t*>(p.expert_x);
  if (p.vec) {
    constexpr int N = Vec16<T>::N;
    for (; item < sh.hi; item += kWarps) {
      const int4 r0 = next[0], r1 = next[1];
      if (item + kWarps < sh.hi) load_piece(item + kWarps);  // ahead of this piece's stores in the memory queue
      const int t = item / P;
      const int v0 = (item - t * P) * p.piece_vecs;
      const int v1 = min(nv, v0 + p.piece_vecs);
      const int32_t* rows = sh.rows + (t - sh.t0) * k;
      float2 y[kLaneVecs][N / 2], acc[kLaneVecs][N / 2];
      float w_lane = 0.f;
      if (FUSED) {
        if (lane < k) w_lane = __ldcg(p.weights + (size_t)t * k + lane);
        expert_output<T>(r0, p.scale, y[0]);
        expert_output<T>(r1, p.scale, y[1]);
#pragma unroll
        for (int e = 0; e < N / 2; ++e) acc[0][e] = acc[1][e] = make_float2(0.f, 0.f);
      }
      const size_t off = ((size_t)v0 + lane) * 16;
      const bool in0 = v0 + lane < v1, in1 = v0 + lane + 32 < v1;
      for (int kk = 0; kk < k; ++kk) {
        const int row = rows[kk];
        const float w = FUSED ? __shfl_sync(0xffffffffu, w_lane, kk) : 0.f;
        if (row < 0) continue;
        int4* d = reinterpret_cast<int4*>(ex + (size_t)row * p.row_bytes + off);
        if (in0) d[0] = r0;
        if (in1) d[32] = r1;
        if (FUSED) {
#pragma unroll
          for (int u = 0; u < kLaneVecs; ++u)
#pragma unroll
            for (int e = 0; e < N / 2; ++e) fma2(acc[u][e], y[u][e], w);
        }
      }
      if (FUSED) {
        int4* o = reinterpret_cast<int4*>(reinterpret_cast<uint8_t*>(p.out) + (size_t)t * p.row_bytes + off);
        if (in0) o[0] = pack_pairs<T>(acc[0]);
        if (in1) o[32] = pack_pairs<T>(acc[1]);
      }
    }
  } else {
    // rows that are not whole aligned 16-byte vectors: element by element
    const int hidden = (int)(p.row_bytes / sizeof(T));
    for (; item < sh.hi; item += kWarps) {  // P == 1: an item is a token
      const T* src = reinterpret_cast<const T*>(p.x) + (size_t)item * hidden;
      const int32_t* rows = sh.rows + (item - sh.t0) * k;
      for (int h = lane; h < hidden; h += 32) {
        const T v = src[h];
        float acc = 0.f;
        const float y = FUSED ? to_f32(from_f32<T>(to_f32(v) * p.scale)) : 0.f;
        for (int kk = 0; kk < k; ++kk) {
          const int row = rows[kk];
          if (row < 0) continue;
          reinterpret_cast<T*>(p.expert_x)[(size_t)row * hidden + h] = v;
          if (FUSED) acc = fmaf(y, __ldcg(p.weights + (size_t)item * k + kk), acc);
        }
        if (FUSED) reinterpret_cast<T*>(p.out)[(size_t)item * hidden + h] = from_f32<T>(acc);
      }
    }
  }
  final_stamps(p, FUSED);
}

// out[t] = sum over k (ascending) of w[t, k] * expert_y[row(t, k)], fp32, rounded once; a token none of whose
// entries was delivered gets a zero row.  One warp per (token, piece of the row).  Eight 16-byte loads per
// lane are in flight whatever k is: KB rows of 8 / KB vectors each.  Bound by the gather of k rows.
template <typename T, int KB>
__global__ void __launch_bounds__(256) moe_local_combine_kernel(const MoeLocalCombineParams p) {
  constexpr int N = Vec16<T>::N;
  constexpr int U = 8 / KB;
  const int lane = threadIdx.x & 31;
  const int k = p.k;
  const int P = p.pieces;
  const int W = (int)(gridDim.x * blockDim.x) >> 5;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  stamp_cta0(p.trace, 0);
  stamp_cta0(p.trace, 1);
  const uint8_t* ey = reinterpret_cast<const uint8_t*>(p.expert_y);
  const int nv = (int)(p.row_bytes >> 4);
  const int items = p.num_tokens * P;
  int item = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int next_row = -1;
  float next_w = 0.f;
  auto ask = [&](int i) {  // route and weights of an item, one iteration ahead of their use
    if (lane < k && i < items) {
      const size_t at = (size_t)(i / P) * k + lane;
      next_row = __ldcg(p.route + at).y;
      next_w = __ldcg(p.weights + at);
    }
  };
  ask(item);
  for (; item < items; item += W) {
    const int t = item / P;
    const int row = next_row;
    const float w = next_w;
    ask(item + W);
    if (p.vec) {
      const int v0 = (item - t * P) * p.piece_vecs;
      const int v1 = min(nv, v0 + p.piece_vecs);
      int4* o = reinterpret_cast<int4*>(reinterpret_cast<uint8_t*>(p.out) + (size_t)t * p.row_bytes);
      for (int vb = v0; vb < v1; vb += 32 * U) {
        float acc[U][N];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int e = 0; e < N; ++e) acc[u][e] = 0.f;
        for (int kb = 0; kb < k; kb += KB) {
          // Every load is unconditional (a lane past the end or an entry that was not delivered reads a valid
          // place and drops the value), so that all of them are issued before the first is used.
          int4 a[KB][U];
#pragma unroll
          for (int q = 0; q < KB; ++q) {
            const int rq = __shfl_sync(0xffffffffu, row, min(kb + q, k - 1));
            const int4* src = reinterpret_cast<const int4*>(ey + (size_t)max(rq, 0) * p.row_bytes);
#pragma unroll
            for (int u = 0; u < U; ++u) a[q][u] = __ldcg(src + min(vb + lane + 32 * u, v1 - 1));
          }
#pragma unroll
          for (int q = 0; q < KB; ++q) {
            const int rq = kb + q < k ? __shfl_sync(0xffffffffu, row, kb + q) : -1;
            const float wq = __shfl_sync(0xffffffffu, w, (kb + q) & 31);
            if (rq < 0) continue;
#pragma unroll
            for (int u = 0; u < U; ++u) fma_vec<T>(acc[u], a[q][u], wq);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int v = vb + lane + 32 * u;
          if (v < v1) o[v] = pack_vec<T>(acc[u]);
        }
      }
    } else {
      const int hidden = (int)(p.row_bytes / sizeof(T));
      for (int h0 = 0; h0 < hidden; h0 += 32) {  // same trip count for every lane: the shuffles need them all
        const int h = h0 + lane;
        float acc = 0.f;
        for (int kk = 0; kk < k; ++kk) {
          const int rq = __shfl_sync(0xffffffffu, row, kk);
          const float wq = __shfl_sync(0xffffffffu, w, kk);
          if (rq >= 0 && h < hidden) acc = fmaf(to_f32(reinterpret_cast<const T*>(p.expert_y)[(size_t)rq * hidden + h]), wq, acc);
        }
        if (h < hidden) reinterpret_cast<T*>(p.out)[(size_t)t * hidden + h] = from_f32<T>(acc);
      }
    }
  }
  stamp_cta0(p.trace, 2);
  stamp_cta0(p.trace, 3);
  stamp_last(p.trace);
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
namespace {

// Pieces of equal size, at most `most` vectors each.
void cut_row(uint32_t row_bytes, bool vec, int most, int32_t* pieces, int32_t* piece_vecs) {
  const int nv = (int)(row_bytes >> 4);
  *pieces = vec ? std::max(1, (nv + most - 1) / most) : 1;
  *piece_vecs = (nv + *pieces - 1) / *pieces;
}

template <typename T>
cudaError_t dispatch_typed(const MoeLocalDispatchParams& p, int threads, int grid, size_t smem, cudaStream_t stream) {
  if (p.out == nullptr) return ptx::launch_dependent(moe_local_dispatch_kernel<T, false, 256>, grid, 256, smem, stream, p);
  if (threads == 256) return ptx::launch_dependent(moe_local_dispatch_kernel<T, true, 256>, grid, 256, smem, stream, p);
  return ptx::launch_dependent(moe_local_dispatch_kernel<T, true, 512>, grid, 512, smem, stream, p);
}

template <typename T>
cudaError_t combine_typed(const MoeLocalCombineParams& p, int grid, cudaStream_t stream) {
  if (p.k <= 2) return ptx::launch_dependent(moe_local_combine_kernel<T, 2>, grid, 256, 0, stream, p);
  if (p.k <= 4) return ptx::launch_dependent(moe_local_combine_kernel<T, 4>, grid, 256, 0, stream, p);
  return ptx::launch_dependent(moe_local_combine_kernel<T, 8>, grid, 256, 0, stream, p);
}

}  // namespace

// A CTA reads the ids of every earlier token, so that work grows with the square of the entries, where the kernel
// with a grid barrier counts every entry once.  The line lies at the most entries that the task's generator draws, the
// range this kernel is tested over; the two do not cross there.  bf16, us, forward / dispatch + combine, on either side:
//   entries                                32768        65536: here, with barrier     131072: here, with barrier
//   64 experts, top-8, rows of 8 KiB     70 / 116     135 / 230      344 / 244        266 / 451      668 / 470
//   256 experts, top-8, rows of 2 KiB    22 / 39       44 / 71       142 / 120         85 / 129      240 / 192
//   64 experts, top-8, rows of 512 B     13 / 18       23 / 34        66 / 55          42 / 71       115 / 95
//   64 experts, top-4, rows of 128 B     14 / 23       24 / 41        82 / 72          44 / 74       139 / 118
// (8192 experts: the counts fill 32 KiB of the 48 KiB of shared memory that need no opt-in.)
bool moe_local_dispatch_applies(int64_t num_entries, int num_experts) {
  return num_entries <= 32768 && num_experts <= 8192;
}

cudaError_t launch_moe_local_dispatch(MoeLocalDispatchParams p, int sms, cudaStream_t stream) {
  if (p.k < 1 || p.k > 32) return cudaErrorInvalidValue;
  p.vec = (p.row_bytes & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 &&
          (reinterpret_cast<uintptr_t>(p.expert_x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
  cut_row(p.row_bytes, p.vec != 0, kPieceVecs, &p.pieces, &p.piece_vecs);
  const int64_t items = (int64_t)p.num_tokens * p.pieces;
  // Plain copies keep the most stores in flight with four CTAs of eight warps per SM (2047 tokens to 16376 rows
  // of 8 KiB: 59 us with combine, 71 with half the warps, 95 with a quarter).  Where the result is formed on the
  // way, the fewer CTAs the less of the counting is repeated: 16 warps per SM (4096 tokens, top-6: 55 us; 57 to
  // 62 with 32 warps), or eight when no warp gets more than two pieces (128 tokens: 6.6 us, 7.2 with 16 warps).
  const bool fused = p.out != nullptr;
  const int threads = fused && items > 16 * (int64_t)sms ? 512 : 256;
  const int warps = threads / 32;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((items + warps - 1) / warps, (int64_t)(fused ? 1 : 4) * sms));
  p.cap = (int32_t)((items + grid - 1) / grid / p.pieces + 2) * p.k;
  p.hist_copies = (p.num_tokens * p.k > 4096 && p.num_experts <= 1024) ? 4 : 1;
  const size_t smem = ((size_t)p.hist_copies * p.num_experts + 2 * (size_t)p.cap) * sizeof(int32_t);
  if (smem > 48 * 1024) return cudaErrorInvalidValue;
  switch (p.dtype) {
    case 0: return dispatch_typed<__half>(p, threads, grid, smem, stream);
    case 1: return dispatch_typed<__nv_bfloat16>(p, threads, grid, smem, stream);
    case 2: return dispatch_typed<float>(p, threads, grid, smem, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_moe_local_combine(MoeLocalCombineParams p, int sms, cudaStream_t stream) {
  if (p.k < 1 || p.k > 32) return cudaErrorInvalidValue;
  if (p.num_tokens == 0) return cudaSuccess;
  p.vec = (p.row_bytes & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.expert_y) & 15u) == 0 &&
          (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
  // 2 KiB pieces when every resident warp (four CTAs of eight per SM) gets one, else 1 KiB ones: 2047 tokens of
  // 8 KiB 58.6 us against 59.7 with dispatch, 3000 of 4000 bytes 17.1 against 18.9, but 300 of 8 KiB 17.0
  // against 13.5.
  const int64_t row_vecs = p.row_bytes >> 4;
  const bool plenty = p.num_tokens * row_vecs >= 2 * kPieceVecs * 32 * (int64_t)sms;
  cut_row(p.row_bytes, p.vec != 0, plenty ? 2 * kPieceVecs : kPieceVecs, &p.pieces, &p.piece_vecs);
  const int64_t warps = (int64_t)p.num_tokens * p.pieces;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, 4 * (int64_t)sms));
  switch (p.dtype) {
    case 0: return combine_typed<__half>(p, grid, stream);
    case 1: return combine_typed<__nv_bfloat16>(p, grid, stream);
    case 2: return combine_typed<float>(p, grid, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace b200
