// MoE dispatch and combine when one rank holds every expert.
//
// With a single rank no row crosses a link, so nothing of the multi-rank protocol is needed: no
// landing buffer, no records for an owner to read back, no flags, no grid barrier.  One ordinary
// launch turns expert ids into slots and writes the rows to their final place; combine gathers them
// by the route table.  The layouts are those of the multi-rank kernels (rows of an expert in
// (token, k) order; 5-int metadata; per-expert counts).
//
// Both kernels may start before the previous kernel of the stream has ended (programmatic dependent launch), so
// what that kernel may have written is read through L2 (ld.global.cg) and only after grid_dep_wait().
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
constexpr int kPieceVecs = 128;            // a warp's share of a row: 2 KiB, four 16-byte vectors per lane
constexpr int kLaneVecs = kPieceVecs / 32;

__device__ __forceinline__ void stamp_cta0(uint64_t* trace, int slot) {
  if (trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0) trace[slot] = global_timer_ns();
}
__device__ __forceinline__ void stamp_last(uint64_t* trace) {
  if (trace != nullptr && threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned long long*>(trace + 7), global_timer_ns());
}

// 16 bytes of T times `s`, rounded to T as the stored expert output would be.
template <typename T>
__device__ __forceinline__ int4 expert_op(const int4& raw, float s) {
  return scale_vec<T>(raw, s);
}

}  // namespace

// Work is T x P items (token, piece of its row); CTA b owns the items [b I / G, (b + 1) I / G) and so the
// tokens they touch.  It counts the entries of all EARLIER tokens per expert by reading their ids itself
// (at most 128 KiB, out of L2) instead of meeting the other CTAs on a barrier, ranks its own entries with
// one warp, and then every warp copies pieces: a piece is read once and stored k times.  Neighbouring CTAs
// may share a token; its metadata belongs to the CTA with its first piece.
//
// FUSED: the caller wants dispatch -> y = x * scale -> combine.  The expert op is elementwise, so its result
// and the weighted sum over the token's k entries are formed from the registers that have just been stored
// to the expert rows; they are not written out and read back.
//
// Bound by the row stores (k per row read).
template <typename T, bool FUSED, int THREADS>
__global__ void __launch_bounds__(THREADS) moe_local_dispatch_kernel(const MoeLocalDispatchParams p) {
  constexpr int kWarps = THREADS / 32;
  extern __shared__ __align__(16) int32_t smem_local[];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int E = p.num_experts;
  const int k = p.k;
  const int P = p.pieces;
  int32_t* s_hist = smem_local;
  int32_t* s_ids = smem_local + E;
  int32_t* s_rows = s_ids + p.cap;

  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  stamp_cta0(p.trace_d, 0);
  const int items = p.num_tokens * P;
  const int lo = (int)((long long)items * blockIdx.x / gridDim.x);
  const int hi = (int)((long long)items * (blockIdx.x + 1) / gridDim.x);
  const int t0 = lo / P;
  const int t1 = (hi + P - 1) / P;
  const int i0 = t0 * k;
  const int m = hi > lo ? t1 * k - i0 : 0;  // own entries

  // the first piece of every warp is on its way while the slots are worked out
  const uint8_t* xb = reinterpret_cast<const uint8_t*>(p.x);
  const int nv = (int)(p.row_bytes >> 4);
  int4 r[kLaneVecs];
  auto load_piece = [&](int item) {
    const int t = item / P;
    const int v0 = (item - t * P) * p.piece_vecs;
    const int v1 = min(nv, v0 + p.piece_vecs);
    const int4* src = reinterpret_cast<const int4*>(xb + (size_t)t * p.row_bytes);
#pragma unroll
    for (int u = 0; u < kLaneVecs; ++u) {
      const int v = v0 + lane + 32 * u;
      if (v < v1) r[u] = __ldcg(src + v);
    }
  };
  int item = lo + warp;
  if (p.vec && item < hi) load_piece(item);

  for (int e = tid; e < E; e += THREADS) s_hist[e] = 0;
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
    auto count = [&](int e) {
      if (e >= 0 && e < E) atomicAdd(&s_hist[e], 1);
    };
    int done = 0;
    if ((reinterpret_cast<uintptr_t>(p.indices) & 15u) == 0) {
      const int4* ids4 = reinterpret_cast<const int4*>(p.indices);
      const int n4 = i0 >> 2;
      constexpr int kFly = 4;  // loads in flight per thread
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
  stamp_cta0(p.trace_d, 1);
  if (warp == 0) {
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
  const int j_lo = ((lo + P - 1) / P) * k - i0;  // entries of tokens whose first piece is this CTA's
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
  if (FUSED) {
    stamp_cta0(p.trace_c, 0);
    stamp_cta0(p.trace_c, 1);
  }

  uint8_t* ex = reinterpret_cast<uint8_t*>(p.expert_x);
  if (p.vec) {
    for (bool first = true; item < hi; item += kWarps, first = false) {
      if (!first) load_piece(item);
      const int t = item / P;
      const int v0 = (item - t * P) * p.piece_vecs;
      const int v1 = min(nv, v0 + p.piece_vecs);
      const int32_t* rows = s_rows + (t - t0) * k;
      for (int kk = 0; kk < k; ++kk) {
        const int row = rows[kk];
        if (row < 0) continue;
        int4* d = reinterpret_cast<int4*>(ex + (size_t)row * p.row_bytes);
#pragma unroll
        for (int u = 0; u < kLaneVecs; ++u) {
          const int v = v0 + lane + 32 * u;
          if (v < v1) d[v] = r[u];
        }
      }
      if (FUSED) {
        constexpr int N = Vec16<T>::N;
        const float w_lane = lane < k ? __ldcg(p.weights + (size_t)t * k + lane) : 0.f;
        int4* o = reinterpret_cast<int4*>(reinterpret_cast<uint8_t*>(p.out) + (size_t)t * p.row_bytes);
#pragma unroll
        for (int u = 0; u < kLaneVecs; ++u) {
          const int v = v0 + lane + 32 * u;
          const int4 y = expert_op<T>(r[u], p.scale);
          float acc[N];
#pragma unroll
          for (int e = 0; e < N; ++e) acc[e] = 0.f;
          for (int kk = 0; kk < k; ++kk) {
            const float w = __shfl_sync(0xffffffffu, w_lane, kk);
            if (rows[kk] >= 0) fma_vec<T>(acc, y, w);
          }
          if (v < v1) o[v] = pack_vec<T>(acc);
        }
      }
    }
  } else {
    // rows that are not whole aligned 16-byte vectors: element by element
    const int hidden = (int)(p.row_bytes / sizeof(T));
    for (; item < hi; item += kWarps) {  // P == 1: an item is a token
      const T* src = reinterpret_cast<const T*>(p.x) + (size_t)item * hidden;
      const int32_t* rows = s_rows + (item - t0) * k;
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
  stamp_cta0(p.trace_d, 6);
  stamp_last(p.trace_d);
  if (FUSED) {
    stamp_cta0(p.trace_c, 2);
    stamp_cta0(p.trace_c, 3);
    stamp_last(p.trace_c);
  }
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
  for (int item = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; item < p.num_tokens * P; item += W) {
    const int t = item / P;
    int row = -1;
    float w = 0.f;
    if (lane < k) {
      row = __ldcg(p.route + (size_t)t * k + lane).y;
      w = __ldcg(p.weights + (size_t)t * k + lane);
    }
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
          int4 a[KB][U];
#pragma unroll
          for (int q = 0; q < KB; ++q) {
            const int rq = kb + q < k ? __shfl_sync(0xffffffffu, row, kb + q) : -1;
            const int4* src = reinterpret_cast<const int4*>(ey + (size_t)rq * p.row_bytes);
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int v = vb + lane + 32 * u;
              a[q][u] = (rq >= 0 && v < v1) ? __ldcg(src + v) : make_int4(0, 0, 0, 0);
            }
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

// Pieces of equal size, at most 2 KiB each.
void cut_row(uint32_t row_bytes, bool vec, int32_t* pieces, int32_t* piece_vecs) {
  const int nv = (int)(row_bytes >> 4);
  *pieces = vec ? std::max(1, (nv + kPieceVecs - 1) / kPieceVecs) : 1;
  *piece_vecs = (nv + *pieces - 1) / *pieces;
}

template <typename T, bool FUSED, int THREADS>
cudaError_t launch_dispatch(const MoeLocalDispatchParams& p, int grid, size_t smem, cudaStream_t stream) {
  return ptx::launch_dependent(moe_local_dispatch_kernel<T, FUSED, THREADS>, grid, THREADS, smem, stream, p);
}

template <typename T>
cudaError_t dispatch_typed(const MoeLocalDispatchParams& p, int grid, int threads, size_t smem, cudaStream_t stream) {
  if (p.out != nullptr)
    return threads == 256 ? launch_dispatch<T, true, 256>(p, grid, smem, stream)
                          : launch_dispatch<T, true, 1024>(p, grid, smem, stream);
  return threads == 256 ? launch_dispatch<T, false, 256>(p, grid, smem, stream)
                        : launch_dispatch<T, false, 1024>(p, grid, smem, stream);
}

template <typename T>
cudaError_t combine_typed(const MoeLocalCombineParams& p, int grid, cudaStream_t stream) {
  if (p.k <= 2) return ptx::launch_dependent(moe_local_combine_kernel<T, 2>, grid, 256, 0, stream, p);
  if (p.k <= 4) return ptx::launch_dependent(moe_local_combine_kernel<T, 4>, grid, 256, 0, stream, p);
  return ptx::launch_dependent(moe_local_combine_kernel<T, 8>, grid, 256, 0, stream, p);
}

}  // namespace

// A CTA reads the ids of every earlier token, so that work grows with the square of the entries; at 32768
// entries it is 128 KiB of L2 reads per SM, a few microseconds beside 200 MB of row stores.  Beyond that the
// kernel with a grid barrier counts every entry once.  (8192 experts: the counts fill 32 KiB of the 48 KiB of
// shared memory that need no opt-in.)
bool moe_local_dispatch_applies(int64_t num_entries, int num_experts) {
  return num_entries <= 32768 && num_experts <= 8192;
}

cudaError_t launch_moe_local_dispatch(MoeLocalDispatchParams p, int sms, cudaStream_t stream) {
  if (p.k < 1 || p.k > 32) return cudaErrorInvalidValue;
  p.vec = (p.row_bytes & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 &&
          (reinterpret_cast<uintptr_t>(p.expert_x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
  cut_row(p.row_bytes, p.vec != 0, &p.pieces, &p.piece_vecs);
  const int items = p.num_tokens * p.pieces;
  // Few entries: CTAs of eight warps, one piece per warp, so that every SM has some of the rows.  Many: one
  // CTA of 32 warps per SM, so that the ids of the earlier tokens are read once per SM.
  const bool small = p.num_tokens * p.k <= 2048;
  const int threads = small ? 256 : 1024;
  const int per_cta = threads / 32;
  const int grid = std::max(1, std::min((items + per_cta - 1) / per_cta, small ? 4 * sms : sms));
  const int items_per_cta = (items + grid - 1) / grid;
  p.cap = (items_per_cta / p.pieces + 2) * p.k;
  const size_t smem = ((size_t)p.num_experts + 2 * (size_t)p.cap) * sizeof(int32_t);
  if (smem > 48 * 1024) return cudaErrorInvalidValue;
  switch (p.dtype) {
    case 0: return dispatch_typed<__half>(p, grid, threads, smem, stream);
    case 1: return dispatch_typed<__nv_bfloat16>(p, grid, threads, smem, stream);
    case 2: return dispatch_typed<float>(p, grid, threads, smem, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_moe_local_combine(MoeLocalCombineParams p, int sms, cudaStream_t stream) {
  if (p.k < 1 || p.k > 32) return cudaErrorInvalidValue;
  if (p.num_tokens == 0) return cudaSuccess;
  p.vec = (p.row_bytes & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.expert_y) & 15u) == 0 &&
          (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
  cut_row(p.row_bytes, p.vec != 0, &p.pieces, &p.piece_vecs);
  const int64_t warps = (int64_t)p.num_tokens * p.pieces;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, 8 * (int64_t)sms));
  switch (p.dtype) {
    case 0: return combine_typed<__half>(p, grid, stream);
    case 1: return combine_typed<__nv_bfloat16>(p, grid, stream);
    case 2: return combine_typed<float>(p, grid, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace b200
