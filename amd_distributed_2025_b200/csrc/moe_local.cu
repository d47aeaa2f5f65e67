// MoE dispatch and combine when one rank holds every expert.
//
// With a single rank no row crosses a link, so nothing of the multi-rank protocol is needed: no
// landing buffer, no records for an owner to read back, no flags, no grid barrier.  One ordinary
// launch turns expert ids into slots and writes the rows to their final place; combine gathers them
// by the route table.  The layouts are those of the multi-rank kernels (rows of an expert in
// (token, k) order; 5-int metadata; per-expert counts).
//
// Both kernels may start before the previous kernel of the stream has ended (programmatic dependent launch): no global
// memory is read or written before grid_dep_wait(), which makes that kernel's stores visible.  Ids, routes, weights and
// whole vectors are read past L1 (ld.global.cg), as nothing comes back for them; ragged rows, element by element, are not.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "moe.h"
#include "moe_common.cuh"
#include "per_device.h"
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

// What a CTA of the dispatch kernel owns: items [lo, hi) and the entries [i0, i0 + m) of the tokens they touch.
struct Share {
  int lo, hi, t0, i0, m;
  int32_t* total;  // shared memory: entries [0, i0 + m) of each expert
  int32_t* ids;    // shared memory: expert of each own entry, or -1; then three words of -2
  int32_t* rows;   // shared memory: final row of each own entry, or -1
};

// Work is T x P items (token, piece of its row), dealt out to the CTAs in runs (moe_runs.h).  Neighbouring CTAs may share
// a token; its metadata belongs to the CTA with its first piece.
__device__ __forceinline__ Share share_of_cta(const MoeLocalDispatchParams& p, int32_t* smem) {
  Share sh;
  const MoeRuns runs(p.num_tokens * p.pieces, (int)gridDim.x, p.slope);
  sh.lo = runs.start((int)blockIdx.x);
  sh.hi = runs.start((int)blockIdx.x + 1);
  sh.t0 = sh.lo / p.pieces;
  sh.i0 = sh.t0 * p.k;
  sh.m = sh.hi > sh.lo ? (sh.hi + p.pieces - 1) / p.pieces * p.k - sh.i0 : 0;
  sh.total = smem;
  sh.ids = smem + ((p.num_experts + 3) & ~3);
  sh.rows = sh.ids + p.cap;
  return sh;
}

// Counts the entries of every expert up to the CTA's last one, by reading the ids itself (at most 128 KiB, out of L2)
// instead of meeting the other CTAs on a barrier, and keeps its own ids.
template <int FLY>
__device__ __forceinline__ void count_entries(const MoeLocalDispatchParams& p, const Share& sh) {
  const int tid = threadIdx.x, threads = blockDim.x;
  auto count = [&](int i, int e) {
    const bool valid = (uint32_t)e < (uint32_t)p.num_experts;
    if (valid) atomicAdd(sh.total + e, 1);
    if (i >= sh.i0) {
      if (!valid) record_status(p.status, STATUS_BAD_INDEX, PHASE_NONE, -1, i, p.epoch, (uint64_t)(int64_t)e);
      sh.ids[i - sh.i0] = valid ? e : -1;
    }
  };
  const int n = sh.i0 + sh.m;
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(p.indices) & 15u) == 0) {
    const int4* ids4 = reinterpret_cast<const int4*>(p.indices);
    const int n4 = n >> 2;
    for (int q0 = tid; q0 < n4; q0 += threads * FLY) {
      int4 a[FLY];  // loads in flight per thread
#pragma unroll
      for (int u = 0; u < FLY; ++u)
        if (q0 + u * threads < n4) a[u] = __ldcg(ids4 + q0 + u * threads);
#pragma unroll
      for (int u = 0; u < FLY; ++u) {
        const int q = q0 + u * threads;
        if (q >= n4) break;
        count(4 * q, a[u].x);
        count(4 * q + 1, a[u].y);
        count(4 * q + 2, a[u].z);
        count(4 * q + 3, a[u].w);
      }
    }
    done = n4 << 2;
  }
  for (int i = done + tid; i < n; i += threads) count(i, __ldcg(p.indices + i));
}

// Final rows of the own entries, a lane each.  An expert's rows are in (token, k) order: the slot of an entry is the
// count up to the CTA's end less the own entries of that expert from it on.
__device__ __forceinline__ void assign_rows(const MoeLocalDispatchParams& p, const Share& sh) {
  const int lane = threadIdx.x & 31;
  for (int j0 = (int)threadIdx.x - lane; j0 < sh.m; j0 += blockDim.x) {
    const int j = j0 + lane;
    const int e = j < sh.m ? sh.ids[j] : -1;
    const int before = e >= 0 ? sh.total[e] : 0;
    int from_here = __popc(__match_any_sync(0xffffffffu, e) & (0xffffffffu << lane));
#pragma unroll 4
    for (int i = j0 + 32; i < sh.m; i += 4) {
      const int4 later = *reinterpret_cast<const int4*>(sh.ids + i);
      from_here += (later.x == e) + (later.y == e) + (later.z == e) + (later.w == e);
    }
    const int slot = before - from_here;
    const bool fits = e >= 0 && slot < p.max_recv;
    if (j < sh.m) sh.rows[j] = fits ? e * p.max_recv + slot : -1;
    // (reported here: the same in the loop that copies rows made forward of 4096 tokens 0.2 us longer)
    if (e >= 0 && !fits) record_status(p.status, STATUS_BAD_INDEX, PHASE_NONE, 0, sh.i0 + j, p.epoch, (uint64_t)slot);
  }
}

// Route table and metadata rows (global expert, source rank, token, k, 0) of a token.
__device__ __forceinline__ void write_metadata(const MoeLocalDispatchParams& p, const Share& sh, int t, int lane) {
  if (lane >= p.k) return;
  const int i = t * p.k + lane;
  const int e = sh.ids[i - sh.i0], row = sh.rows[i - sh.i0];
  p.route[i] = make_int2(row >= 0 ? 0 : -1, row);
  if (row >= 0) {
    int32_t* meta = p.expert_meta + (size_t)row * kMetaDim;
    meta[0] = e;
    meta[1] = 0;
    meta[2] = t;
    meta[3] = lane;
    meta[4] = 0;
  }
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
// stores: 268 MB (4096 tokens, top-6, hidden 4096) in 52 us, where a bare copy of the same pattern takes 48 to
// 51.  Moving the pieces through shared memory with bulk copies measured 53 us there but 67 us (against 59)
// for dispatch + combine of 2047 tokens.
//
// Small ones are bound by latency.  Index arithmetic and zeroing run before grid_dep_wait(), beside the previous
// kernel; then all loads (ids of earlier and own entries, the first row piece, its weights) leave together, so that one
// memory latency lies before the first store, and ranks come from one warp match.  With own ids, earlier ids and weights
// asked for one after the other, and one warp ranking 32 entries at a time: 11 tokens, top-2 4.4 us in a graph, now 3.1;
// 128 tokens, top-8, 256 experts 6.6, now 5.1; 101 tokens, top-4 4.2, now 3.3; 32 tokens, rows of 1 KiB 3.8, now 2.7.
// Ranks worked out by every warp for itself cost 8.8 us at 128 tokens, clusters that share the counting 5.2 (pairs, and
// nothing for plain copies) to 8.4 (eight CTAs), L2 prefetches before the wait changed nothing, and neither did
// stores with an evict-first policy.
template <typename T, bool FUSED>
__global__ void __launch_bounds__(FUSED ? 512 : 1024, 1) moe_local_dispatch_kernel(const MoeLocalDispatchParams p) {
  constexpr int kLaneVecs = kPieceVecs / 32;
  static_assert(kLaneVecs == 2, "the copy loop is written for two vectors per lane");
  extern __shared__ __align__(128) uint8_t smem_local[];
  const int lane = threadIdx.x & 31;
  const int threads = blockDim.x, warps = threads >> 5;
  const int k = p.k;
  const int P = p.pieces;
  const Share sh = share_of_cta(p, reinterpret_cast<int32_t*>(smem_local));
  for (int i = threadIdx.x; i < (int)(sh.ids - sh.total); i += threads) sh.total[i] = 0;
  if (threadIdx.x < 3) sh.ids[sh.m + threadIdx.x] = -2;
  const int nv = (int)(p.row_bytes >> 4);
  int item = sh.lo + (int)(threadIdx.x >> 5);
  int4 next[kLaneVecs];
  float next_w = 0.f;
  auto load_piece = [&](int item) {
    const int t = item / P;
    const int v0 = (item - t * P) * p.piece_vecs;
    const int v1 = min(nv, v0 + p.piece_vecs);
    const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(p.x) + (size_t)t * p.row_bytes);
#pragma unroll
    for (int u = 0; u < kLaneVecs; ++u)
      if (v0 + lane + 32 * u < v1) next[u] = __ldcg(src + v0 + lane + 32 * u);
    if (FUSED && lane < k) next_w = __ldcg(p.weights + (size_t)t * k + lane);
  };
  __syncthreads();
  ptx::grid_dep_wait();
  stamp_cta0(p.trace_d, 0);
  if (p.vec && item < sh.hi) load_piece(item);
  count_entries<4>(p, sh);
  __syncthreads();
  stamp_cta0(p.trace_d, 1);
  assign_rows(p, sh);
  __syncthreads();
  stamp_cta0(p.trace_d, 2);
  if (blockIdx.x == gridDim.x - 1) {
    for (int e = threadIdx.x; e < p.num_experts; e += threads)
      p.expert_num_tokens[e] = min(sh.total[e], p.max_recv);
  }
  stamp_cta0(p.trace_d, 3);
  stamp_cta0(p.trace_d, 4);
  stamp_cta0(p.trace_d, 5);
  if (FUSED) {
    stamp_cta0(p.trace_c, 0);
    stamp_cta0(p.trace_c, 1);
  }
  // The next launch is let in when the stores begin (its CTAs would only stand in line for the SMs before: 0.1 us); behind
  // plain copies, combine as a rule, not before the CTAs leave: several of its CTAs fit on an SM, and early ones gather
  // where a dispatch CTA has just left (111 tokens, top-7, 2 KiB, dispatch + combine 8.1 us, now 6.9; 2000, top-2, 2 KiB
  // 8.2, now 7.8).
  if (FUSED) ptx::grid_dep_launch();
  uint8_t* ex = reinterpret_cast<uint8_t*>(p.expert_x);
  if (p.vec) {
    constexpr int N = Vec16<T>::N;
    for (; item < sh.hi; item += warps) {
      const int4 r0 = next[0], r1 = next[1];
      const float w_lane = next_w;
      if (item + warps < sh.hi) load_piece(item + warps);  // ahead of this piece's stores in the memory queue
      const int t = item / P;
      const int piece = item - t * P;
      const int v0 = piece * p.piece_vecs;
      const int v1 = min(nv, v0 + p.piece_vecs);
      const int32_t* rows = sh.rows + (t - sh.t0) * k;
      if (piece == 0) write_metadata(p, sh, t, lane);
      float2 y[kLaneVecs][N / 2], acc[kLaneVecs][N / 2];
      if (FUSED) {
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
    for (; item < sh.hi; item += warps) {  // P == 1: an item is a token
      const T* src = reinterpret_cast<const T*>(p.x) + (size_t)item * hidden;
      const int32_t* rows = sh.rows + (item - sh.t0) * k;
      const float w_lane = FUSED && lane < k ? __ldcg(p.weights + (size_t)item * k + lane) : 0.f;
      write_metadata(p, sh, item, lane);
      for (int h0 = 0; h0 < hidden; h0 += 32) {  // same trip count for every lane: the shuffles need them all
        const int h = h0 + lane;
        const bool in = h < hidden;
        const T v = in ? src[h] : from_f32<T>(0.f);
        float acc = 0.f;
        const float y = FUSED ? to_f32(from_f32<T>(to_f32(v) * p.scale)) : 0.f;
        for (int kk = 0; kk < k; ++kk) {
          const int row = rows[kk];
          const float w = FUSED ? __shfl_sync(0xffffffffu, w_lane, kk) : 0.f;
          if (row < 0) continue;
          if (in) reinterpret_cast<T*>(p.expert_x)[(size_t)row * hidden + h] = v;
          if (FUSED) acc = fmaf(y, w, acc);
        }
        if (FUSED && in) reinterpret_cast<T*>(p.out)[(size_t)item * hidden + h] = from_f32<T>(acc);
      }
    }
  }
  final_stamps(p, FUSED);
}

// out[t] = sum over k (ascending) of w[t, k] * expert_y[row(t, k)], fp32, rounded once; a token none of whose
// entries was delivered gets a zero row.  One warp per (token, piece of the row), 1 KiB of KB rows at a
// time: KB is k, or k in equal rounds (the launcher says of how many at most).  Bound by the gather of k rows.  What counts
// is that a request is 1 KiB of a row and that no round is partly idle, not how many loads a lane has in flight: eight
// whatever k is, as 512 bytes of eight rows or 2 KiB of two, took (combine alone, rows in L2, us) 8.1 at 600 tokens, top-8,
// rows of 8 KiB, now 6.9; 9.8 at 1500, top-6, 4 KiB, now 7.4; 4.4 at 4000, top-2, 1 KiB, now 3.2; 6.2 at 1000, top-3,
// 8 KiB, now 5.7.
template <typename T, int KB>
__global__ void __launch_bounds__(256) moe_local_combine_kernel(const MoeLocalCombineParams p) {
  constexpr int N = Vec16<T>::N;
  constexpr int U = 2;
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
          const T* src = reinterpret_cast<const T*>(p.expert_y) + (size_t)max(rq, 0) * hidden;
          if (rq >= 0 && h < hidden) acc = fmaf(to_f32(src[h]), wq, acc);
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

// Shared memory that keeps a CTA of forward alone on its SM.  A launch of one CTA per SM starts while the one before it
// still runs; where two fit, the scheduler may put two on each SM that happens to be free, none on the others, and the next
// launch into the gaps, call after call: 128 tokens, top-8 took 7.05 us in a row of calls, 5.3 with one CTA to an SM (129
// and 136 likewise, 140 never).  What that costs: beside a kernel on another stream that holds most of the shared memory,
// forward waits for whole SMs (beside a library GEMM of 4096^3, us a call: 128 tokens 26, two CTAs to an SM 9; 11 tokens
// 4.7 and 4.4; 1000 tokens of 4 KiB 27 either way; beside an elementwise kernel over 512 MB 25 either way).  The other
// remedy, to let the next launch in only when the CTAs leave, costs a row of calls less than 0.1 us at 128 tokens, but 2 to
// 7 % in a graph and at most sizes.
constexpr int kAloneBytes = 116 * 1024;

template <typename T>
cudaError_t dispatch_typed(const MoeLocalDispatchParams& p, int threads, int grid, size_t smem, cudaStream_t stream) {
  if (p.out == nullptr) return ptx::launch_dependent(moe_local_dispatch_kernel<T, false>, grid, threads, smem, stream, p);
  static OncePerDevice once;
  const cudaError_t opted = once([] { return opt_in(moe_local_dispatch_kernel<T, true>, kAloneBytes, false); });
  if (opted != cudaSuccess) return opted;
  const size_t alone = std::max<size_t>(smem, kAloneBytes);
  return ptx::launch_dependent(moe_local_dispatch_kernel<T, true>, grid, threads, alone, stream, p);
}

template <typename T>
cudaError_t combine_typed(const MoeLocalCombineParams& p, int grid, int most, cudaStream_t stream) {
  const int rounds = (p.k + most - 1) / most;
  switch ((p.k + rounds - 1) / rounds) {
    case 1: return ptx::launch_dependent(moe_local_combine_kernel<T, 1>, grid, 256, 0, stream, p);
    case 2: return ptx::launch_dependent(moe_local_combine_kernel<T, 2>, grid, 256, 0, stream, p);
    case 3: return ptx::launch_dependent(moe_local_combine_kernel<T, 3>, grid, 256, 0, stream, p);
    default: return ptx::launch_dependent(moe_local_combine_kernel<T, 4>, grid, 256, 0, stream, p);
  }
}

}  // namespace

// A CTA reads the ids of every earlier token, so that work grows with the square of the entries, where the kernel
// with a grid barrier counts every entry once.  The line lies at the most entries that the task's generator draws, the
// range this kernel is tested over, and beyond which forward() writes expert_y; the two do not cross there, nor at four
// times as many.  bf16, us, forward / dispatch + combine, this kernel and the one with the barrier:
//   entries                                 32768                  65536                  131072
//   64 experts, top-8, rows of 8 KiB    66/111  194/152       133/225  340/241       265/437  651/454
//   256 experts, top-8, rows of 2 KiB   19/36    96/85         40/64   143/120        85/121  235/191
//   64 experts, top-8, rows of 512 B    11/16    47/42         19/29    68/57         41/57   119/99
//   64 experts, top-4, rows of 128 B    12/16    52/47         21/26    78/68         41/49   135/114
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
  if (items > INT32_MAX) return cudaErrorInvalidValue;  // (2 TB of rows)
  // 32 warps per SM keep the most stores in flight where rows are only copied (2047 tokens to 16376 rows of 8 KiB: 30 us,
  // 44 with half the warps).  Every CTA counts for itself, so few large ones repeat less of that: it pays from some
  // 6000 entries on (4000 tokens, top-2, rows of 1 KiB, with combine: 9.2 us with 2 x 16 warps, 10.0 with 4 x 8; 606 items
  // 6.6 and 5.6).  Where the result is formed on the way there is one CTA per SM: 16 warps when each gets more than one
  // piece (4096 tokens, top-6, rows of 8 KiB: 52 us; 58 to 60 with 32 warps), eight when that is two rounds or less
  // (128 tokens, 12 pieces per SM: 5.3 us, 6.0 with 16 warps), ten in between (us with 8, 10 and 16 warps: 300 tokens, 16
  // pieces, 6.1, 5.6, 6.0; 180 tokens, 17 pieces, 7.4, 6.8, 7.3; 600 tokens, 16 pieces, 4.9, 4.3, 4.7; but at the ends of
  // the range 520 tokens, 14 pieces, 4.5, 4.3, 4.1 and 740 tokens, 20 pieces, 5.2, 5.0, 4.7).
  const bool fused = p.out != nullptr;
  const int64_t entries = (int64_t)p.num_tokens * p.k;
  const int threads = !fused ? (entries > 6144 ? 512 : 256)
                             : (items > 20 * (int64_t)sms ? 512 : items > 14 * (int64_t)sms ? 320 : 256);
  const int warps = threads / 32;
  const int ctas = fused ? sms : (32 / warps) * sms;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((items + warps - 1) / warps, ctas));
  // The later a CTA's tokens, the longer it counts before its first store.  With three entries a token and more, a tenth
  // evens that out (4096 tokens, top-6, rows of 8 KiB: 55.5 us without, 53.0 with, 54.7 with two tenths; 2000, top-4, 8 KiB
  // 17.8, 17.5, 18.1; 1500, top-3, 8 KiB 12.3, 11.8; but 1500, top-3, 14 KiB 18.8, 19.3), two tenths where counting is long
  // against the stores (4096, top-8, 1 KiB 13.6, 13.2, 12.4; 4096, top-8, 512 bytes 11.0, 10.9, 10.5; between the two, 2000,
  // top-8, 2 KiB 10.8, 10.4, 10.0).  With one or two, nothing on the average of 36 sizes, and up to 7 % lost (800 tokens,
  // top-1, 14 KiB 7.3 without, 7.8 with a tenth; 1500, top-2, 14 KiB 15.1, 15.6; 3000, top-2, 4 KiB 10.6, 10.3).
  const double lean = !fused || threads < 512 || p.k < 3 ? 0.0 : entries > 16384 && p.row_bytes <= 2048 ? 0.2 : 0.1;
  p.slope = moe_run_slope((int32_t)items, grid, lean);
  const int32_t longest = MoeRuns((int32_t)items, grid, p.slope).longest();
  p.cap = (int32_t)(moe_run_entries(longest, p.pieces, p.k) + 6) & ~3;  // (and three words, in groups of four)
  const size_t smem = ((size_t)((p.num_experts + 3) & ~3) + 2 * (size_t)p.cap) * sizeof(int32_t);
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
  // What counts is how full the last round of the resident warps (four CTAs of eight per SM) is, and how many dependent
  // loads an item takes: few where there is about one item a warp, many short items where there are several.
  // Up to three entries a token, gathered at once: 2 KiB pieces as soon as every warp gets one (2250 tokens, top-1, rows
  // of 8 KiB 5.6 us against 6.2 with 1 KiB ones, top-3 9.9 and 11.0; but 1599, top-3 9.1 and 8.2).
  // More of them: 1 KiB pieces, and rows two at a time from 1.75 items a warp on, else up to four (us, two / up to four):
  //   items a warp                     1.4          1.7          1.85         2.0          2.7          6
  //   top-4, rows of 14 KiB        6.3 / 5.8    6.4 / 6.6    6.5 / 7.5    6.5 / 8.0    9.5 / 10.6   34.2 / 40.6
  //   top-7, rows of 8 KiB         9.5 / 8.2   10.0 / 9.8   10.4 / 12.2  10.6 / 13.2  14.7 / 15.5  41.6 / 47.8
  //   top-8, rows of 5760 bytes   10.3 / 8.8   10.7 / 12.4  11.4 / 14.4  14.2 / 15.5  18.0 / 18.2  45.5 / 53.2
  // (Combine alone; with dispatch before it, 623 tokens, top-8, rows of 14 KiB 32.3 and 35.6.  2 KiB pieces of three rows at
  // a time, as from two items a warp on before: 779 of these tokens 42.5, this way 40.0; 2724 tokens, top-12, rows of 4 KiB
  // 62.3, 60.0; 1185, top-4, 14 KiB 32.8, 33.2; of 80 counts of tokens they are ahead at 22, by 2 % at most.)
  const int64_t resident = 32 * (int64_t)sms;
  cut_row(p.row_bytes, p.vec != 0, kPieceVecs, &p.pieces, &p.piece_vecs);
  if (p.k <= 3 && p.num_tokens * (int64_t)(p.row_bytes >> 4) >= 2 * kPieceVecs * resident)
    cut_row(p.row_bytes, p.vec != 0, 2 * kPieceVecs, &p.pieces, &p.piece_vecs);
  const int most = p.k > 3 && 4 * (int64_t)p.num_tokens * p.pieces >= 7 * resident ? 2 : 4;
  const int64_t warps = (int64_t)p.num_tokens * p.pieces;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, 4 * (int64_t)sms));
  switch (p.dtype) {
    case 0: return combine_typed<__half>(p, grid, most, stream);
    case 1: return combine_typed<__nv_bfloat16>(p, grid, most, stream);
    case 2: return combine_typed<float>(p, grid, most, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace b200
