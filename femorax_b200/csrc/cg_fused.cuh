// One Jacobi-PCG iteration's vector work in one cooperative launch: p.Ap, alpha, the updates of x and
// r, r.r and r.z, the convergence test, beta and the update of p, for solves whose chunks all fit on
// the GPU at once (a block of 256 threads per 2048-entry chunk). The blocks of one solve meet twice,
// at the two reductions; the chunk's p, Ap, then z and r stay in shared memory and its x, r and
// inverse diagonal in registers in between, so every vector is read once and written once.
//
// The sums are those of the separate kernels, in their order (vector.hpp: a warp per chunk in lane
// order, then the chunk sums in lane order; every block forms the second level for itself), so an
// iteration gives the same bits whichever form runs.
//
// What bounds it is latency, about 10 us a launch from 9 to 131 chunks and 13 us at 516 (FP32): the
// chains of dependent additions the documented order needs (64 per lane and 32 over the lanes, then
// the chunk sums, twice; 10.6 cycles each), the two meetings (1.1 us each), the first loads and the
// instruction fetches. As separate kernels (p.Ap, update, p, each with its launch, its loads and its
// last block's levels) they took 20 us; B200, with the operator: an iteration of the 32^3 cube's solve
// 31.6 -> 17.3 us (box tiles shortened too), the batched J2 columns' load step 52.7 -> 40 ms, 16 served
// static solves 82 -> 65 ms.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"
#include "vector.hpp"

namespace fx {
namespace cgf {

// Polls of a meeting before a block gives up (a second or more) unless the caller sets another limit:
// every block of the launch is resident, so a meeting ends as soon as the slowest block has summed its
// chunk.
constexpr int kPolls = 1 << 22;

enum : int { kGoOn = 0, kConverged, kLimit, kIndefinite, kGaveUp };

// Arrives at the meeting counted by *cnt (one thread; its own earlier writes are seen by every thread
// that the meeting releases): the count at which all n arrivals of this meeting are in. The counter
// only grows, n per meeting, so it needs no reset between launches.
__device__ __forceinline__ unsigned long long arrive(unsigned long long* cnt, unsigned n) {
  unsigned long long ticket;
  asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], 1;" : "=l"(ticket) : "l"(cnt) : "memory");
  const unsigned rest = ticket >> 32 ? static_cast<unsigned>(ticket % n) : static_cast<unsigned>(ticket) % n;
  return ticket + (n - rest);
}
// Waits until the count is reached; false when it gives up.
__device__ __forceinline__ bool wait(unsigned long long* cnt, unsigned long long target, int polls) {
  unsigned long long now;
  for (int i = 0; i < polls; ++i) {
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(cnt) : "memory");
    if (now >= target) return true;
  }
  return false;
}

// The lanes' sums added in lane order, in every lane.
__device__ __forceinline__ double lane_sum(double acc, int lanes) {
  double total = 0.0;
#pragma unroll 8
  for (int j = 0; j < lanes; ++j) total += __shfl_sync(0xffffffffu, acc, j);
  return total;
}

// chunk_fma_sum of a chunk whose entries past `len` are zeros (which change no sum: a lane's sum is
// never -0): with 32 lanes all kChunk / 32 terms of a lane, 16 loaded ahead of their additions.
template <class T>
__device__ __forceinline__ double chunk_sum(const T* a, const T* b, int len, int lanes, int lane) {
  if (lanes != 32) return chunk_fma_sum(a, b, len, lanes, lane);
  constexpr int U = 16;
  double acc = 0.0;
#pragma unroll 1
  for (int k = 0; k < kChunk / 32; k += U) {
    T va[U], vb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      va[u] = a[lane + 32 * (k + u)];
      vb[u] = b[lane + 32 * (k + u)];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) acc = fma(static_cast<double>(va[u]), static_cast<double>(vb[u]), acc);
  }
  return lane_sum(acc, lanes);
}

// The second level over nc <= 2048 chunk sums (k_reduce_chunks' order), by one warp, through L2: 8
// loads of a lane ahead of their additions (zeros past the last).
__device__ __forceinline__ double level(const double* part, int nc, int lanes, int lane) {
  constexpr int U = 8;
  double acc = 0.0;
  if (lane < lanes)
    for (int k = lane; k < nc; k += U * lanes) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = k + u * lanes < nc ? __ldcg(part + k + u * lanes) : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) acc += v[u];
    }
  return lane_sum(acc, lanes);
}

template <class T>
struct Chunk {
  T* p;
  const T* ap;
  const T* inv;
  T* x;
  T* r;
  int64_t begin;   // the chunk's first entry
  int len, lanes;
  int64_t c, nc;   // the chunk's place among the solve's chunks
  double* part;    // the solve's chunk sums: p.Ap, r.r and r.z, `ld` apart
  int64_t ld;
  unsigned long long* bar;  // the solve's two meetings
  double rz, tol;
  int it, max_it;  // iterations done so far, and their limit
  int polls;       // of a meeting before a block gives up
};
struct Sums {
  double pap, rr, rz;
  int state;
};

template <class T>
struct Pair;
template <>
struct Pair<double> {
  using type = double2;
};
template <>
struct Pair<float> {
  using type = float2;
};

// A thread's entries of a chunk are the pairs 2 (t + 256 k), k < kPairs; zeros past the chunk's end.
constexpr int kPairs = kChunkPer / 2;
__device__ __forceinline__ int pair_at(int k) { return 2 * (static_cast<int>(threadIdx.x) + k * kChunkBlock); }
template <class T>
__device__ __forceinline__ void load_pairs(const T* v, int len, T (&out)[kChunkPer]) {
#pragma unroll
  for (int k = 0; k < kPairs; ++k) {
    const int j = pair_at(k);
    typename Pair<T>::type q{T(0), T(0)};
    if (j + 1 < len) q = *reinterpret_cast<const typename Pair<T>::type*>(v + j);
    else if (j < len) q.x = v[j];
    out[2 * k] = q.x;
    out[2 * k + 1] = q.y;
  }
}
template <class T>
__device__ __forceinline__ void store_pairs(T* v, int len, const T (&in)[kChunkPer]) {
#pragma unroll
  for (int k = 0; k < kPairs; ++k) {
    const int j = pair_at(k);
    if (j + 1 < len) *reinterpret_cast<typename Pair<T>::type*>(v + j) = {in[2 * k], in[2 * k + 1]};
    else if (j < len) v[j] = in[2 * k];
  }
}

// The iteration of this block's chunk (all 256 threads); the sums and the state are the same in every
// thread of every block of the solve. The solver's vectors are aligned to pairs. The two reductions are two turns of one loop: straight-line code that
// runs once per launch costs more in instruction fetches than in issue.
template <class T>
__device__ __forceinline__ Sums iterate(const Chunk<T>& a) {
  __shared__ __align__(16) T sa[kChunk], sb[kChunk];  // p then z, Ap then r
  __shared__ double sum[3];
  __shared__ int met[3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T vp[kChunkPer], vi[kChunkPer], vr[kChunkPer], vx[kChunkPer];
  load_pairs(a.p + a.begin, a.len, vp);
  load_pairs(a.ap + a.begin, a.len, vi);
  store_pairs(sa, kChunk, vp);
  store_pairs(sb, kChunk, vi);
  Sums o{0.0, 0.0, 0.0, kGoOn};
#pragma unroll 1
  for (int turn = 0; turn < 2; ++turn) {
    if (turn == 1) {  // alpha, x, r and z
      const T alpha = static_cast<T>(a.rz / o.pap);
      T va[kChunkPer];
      load_pairs(sa, kChunk, vp);
      load_pairs(sb, kChunk, va);
#pragma unroll
      for (int k = 0; k < kChunkPer; ++k) {
        vx[k] = fma(alpha, vp[k], vx[k]);
        vr[k] = fma(-alpha, va[k], vr[k]);
        vi[k] = vi[k] * vr[k];
      }
      if (!(fabs(alpha) < INFINITY))  // (it made NaN of the zeros past the chunk's end)
#pragma unroll
        for (int k = 0; k < kChunkPer; ++k)
          if (pair_at(k / 2) + k % 2 >= a.len) vr[k] = vi[k] = T(0);
      store_pairs(sb, kChunk, vr);
      store_pairs(sa, kChunk, vi);
    }
    __syncthreads();
    double* col = a.part + (turn + warp) * a.ld;
    unsigned long long target = 0;
    if (warp <= turn) {  // p.Ap; then r.r and r.z, a warp each
      const double s = chunk_sum(turn == 0 ? sa : sb, turn == warp ? (turn == 0 ? sb : sa) : sb, a.len, a.lanes, lane);
      if (lane == 0) {
        col[a.c] = s;
        if (a.nc > 1) target = arrive(&a.bar[turn], static_cast<unsigned>((turn + 1) * a.nc));
      }
    }
    // Between the arrival and the wait, so that the arrival's release has no other access of its thread
    // to wait for (7.5 us each where these came first)
    if (turn == 0) {
      load_pairs(a.r + a.begin, a.len, vr);
      load_pairs(a.inv + a.begin, a.len, vi);
#pragma unroll
      for (int k = 0; k < kChunkPer; ++k) {
        const int j = pair_at(k / 2) + k % 2;
        vx[k] = j < a.len ? a.x[a.begin + j] : T(0);
      }
    } else {
      store_pairs(a.r + a.begin, a.len, vr);
#pragma unroll
      for (int k = 0; k < kChunkPer; ++k) {
        const int j = pair_at(k / 2) + k % 2;
        if (j < a.len) a.x[a.begin + j] = vx[k];
      }
    }
    if (warp <= turn) {
      if (lane == 0) met[turn + warp] = a.nc == 1 || wait(&a.bar[turn], target, a.polls);
      __syncwarp();
      const double s = level(col, static_cast<int>(a.nc), a.lanes, lane);
      if (lane == 0) sum[turn + warp] = s;
    }
    __syncthreads();
    if (!met[turn] || !met[2 * turn]) {
      o.state = kGaveUp;
      return o;
    }
    if (turn == 0) {
      o.pap = sum[0];
      if (!(o.pap > 0.0)) {
        o.state = kIndefinite;
        return o;
      }
    }
  }
  o.rr = sum[1];
  o.rz = sum[2];
  if (sqrt(o.rr) <= a.tol) {
    o.state = kConverged;
    return o;
  }
  if (a.it + 1 >= a.max_it) {
    o.state = kLimit;
    return o;
  }
  const T beta = static_cast<T>(o.rz / a.rz);
#pragma unroll
  for (int k = 0; k < kChunkPer; ++k) vp[k] = fma(beta, vp[k], vi[k]);
  store_pairs(a.p + a.begin, a.len, vp);
  return o;
}

// CTAs per SM the register budgets are sized for: a chunk's x, r, inverse diagonal and p in registers
template <class T>
constexpr int kMinBlocks = sizeof(T) == 8 ? 2 : 4;

// Chunks (blocks) that fit on the current device at once for kernel `kern` (`known`: a static of the
// launch site).
template <class Kernel>
int64_t capacity(PerDevice<int64_t>& known, Kernel kern) {
  return known.get(current_device(), [&] {
    int per_sm = 0;
    FX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kChunkBlock, 0));
    return static_cast<int64_t>(per_sm) * num_sms();
  });
}

// A cooperative launch of `blocks` blocks (all resident together, or the launch fails).
template <class... Params, class... Args>
void launch(void (*kern)(Params...), int64_t blocks, cudaStream_t st, Args... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(kChunkBlock);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  FX_CUDA(cudaLaunchKernelEx(&cfg, kern, Params(args)...));
}

}  // namespace cgf
}  // namespace fx
