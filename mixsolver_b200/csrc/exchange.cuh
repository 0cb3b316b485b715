// exchange.cuh -- values and sums that the blocks of a resident solve exchange
// through global memory without a barrier: each 8-byte word carries 32 bits of
// the value and the number of its exchange, so the data is its own signal (the
// words are written and read by relaxed 64-bit accesses, which are single-copy
// atomic).
#pragma once

#include "persist.cuh"

namespace mgpu {
namespace {

extern __shared__ __align__(16) unsigned char block_smem[];  // a resident block's dynamic shared memory

template <typename T>
__device__ __forceinline__ T& smem_at(int base, int i) {
  return reinterpret_cast<T*>(block_smem + base)[i];
}

using u64 = unsigned long long;

// Exchange words: value in the low half, exchange number in the high half.
__device__ __forceinline__ u64 pack_word(unsigned v, unsigned seq) { return ((u64)seq << 32) | v; }
__device__ __forceinline__ void st_word(u64* p, u64 v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ u64 ld_word(const u64* p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// A double as two exchange words (its halves), 16-byte aligned.
__device__ __forceinline__ void st_pair(u64* p, double d, unsigned seq) {
  const u64 b = (u64)__double_as_longlong(d);
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(pack_word((unsigned)b, seq)),
               "l"(pack_word((unsigned)(b >> 32), seq))
               : "memory");
}
__device__ __forceinline__ void ld_pair(const u64* p, u64& a, u64& b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

// Failed polls before a wait for other blocks gives up, ~2 s: each is a trip to
// L2, or a shared-memory load where another warp of the block brings the value.
constexpr unsigned kHaloSpins = 1u << 22;
constexpr unsigned kSharedSpins = 1u << 26;

// The limits of a launch, kernel arguments: the sums' barrier takes the spin_limit
// tuning key, values take exchange_spin_limit. Polls follow one another at once:
// with the limits in shared memory and the sleep of vg_sync (barrier_poll_ns)
// between the barrier's polls a pass of the 42,253-row channel took 4.67 ms, 4.56 so.
struct WaitLimits {
  unsigned barrier, value, shared;
};
__host__ __device__ constexpr WaitLimits wait_limits(unsigned spin_limit, unsigned exchange_limit) {
  return {spin_limit ? spin_limit : kHaloSpins, exchange_limit ? exchange_limit : kHaloSpins,
          exchange_limit ? exchange_limit : kSharedSpins};
}

// One more failed poll of a wait, of the polls left: false once none is or another
// block has flagged a timeout.
__device__ __forceinline__ bool keep_polling(unsigned& left, DevStatus* st) {
  if ((--left & 1023u) == 0u && (left == 0u || ld_acquire_i32(&st->timeout) != 0)) {
    atomicExch(&st->timeout, 1);
    return false;
  }
  return true;
}

// This thread's value c[q] of its row in tile k (rows k * blockDim.x ... of the
// block's range) into the chunk sums: a butterfly over the 32 rows of a warp.
template <int NQ>
__device__ __forceinline__ void resident_put(int cp, int cps, int k, const double (&c)[NQ]) {
  double s[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) s[q] = warp_sum(c[q]);
  if ((threadIdx.x & 31) == 0) {
    const int slot = k * (blockDim.x >> 5) + (threadIdx.x >> 5);
#pragma unroll
    for (int q = 0; q < NQ; ++q) smem_at<double>(cp, q * cps + slot) = s[q];
  }
}

constexpr int kSumGroups = 64;  // groups of 256 super-chunks (65,536 rows) of a system, at most
__shared__ double s_group[2][2][kSumGroups];  // group sums: half, sum, group

// The group barrier in two halves, so that other work can run while the
// arrivals travel: what the block wrote before arrive is visible to every
// block after its wait (release and acquire on the counter, as in vg_sync).
__device__ __forceinline__ void vg_arrive(const VGrid& g) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(g.bar) : "memory");
}

__device__ __forceinline__ bool vg_wait(VGrid& g, unsigned limit, DevStatus* st) {
  bool ok = true;
  if (threadIdx.x == 0) {
    unsigned left = limit;
    while (ok && ld_acquire_u64(g.bar) < g.next) ok = keep_polling(left, st);
  }
  g.next += (u64)g.nb;
  return __syncthreads_and(ok) != 0;
}

// The layout-independent sum over all rows (the 32 rows of a chunk in a
// butterfly, the 8 chunk sums of a 256-row super-chunk in order, super-chunks l,
// l + 32, ... of a group of 256 in order, the 32 lane sums in a butterfly, the
// group sums in order), as an arrival and a wait: total_post (every thread,
// after the chunk sums are put) writes this block's super-chunk sums,
// total_wait forms the total. The sums alternate between two halves: a block
// writes sum s + 2 after the barrier of s + 1, at which every block has read
// all of s.

// The super-chunk sums of the state's rows (every thread; the chunk sums are
// read only before the closing barrier of whoever puts the next ones).
template <int NQ, typename State>
__device__ __forceinline__ void super_sums(const State& S) {
  constexpr int kChunks = kSuperRows / 32;
  double* sums = S.sums + (S.rseq & 1u) * 2l * S.nsc;
  __syncthreads();  // the chunk sums are written
  const int first = S.start / kSuperRows, mine = (S.end - S.start + kSuperRows - 1) / kSuperRows;
  for (int j = threadIdx.x; j < mine * NQ; j += blockDim.x) {
    const int q = NQ == 1 ? 0 : j & 1, b = NQ == 1 ? j : j >> 1;
    const double* cq = &smem_at<double>(S.cp, q * S.cps + b * kChunks);
    double acc = cq[0];
#pragma unroll
    for (int c = 1; c < kChunks; ++c) acc = acc + cq[c];
    sums[(long)q * S.nsc + first + b] = acc;
  }
}

template <int NQ, typename State>
__device__ __forceinline__ void total_post(State& S, const VGrid& g) {
  ++S.rseq;
  super_sums<NQ>(S);
  vg_arrive(g);
}

template <int NQ, typename State>
__device__ __forceinline__ bool total_wait(State& S, VGrid& g, DevStatus* st, double (&out)[NQ]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned half = S.rseq & 1u;
  const int nsc = S.nsc, ng = (nsc + 255) >> 8;
  const double* sums = S.sums + half * 2l * nsc;
  if (!vg_wait(g, S.waits.barrier, st)) return false;
  for (int k = warp; k < ng * NQ; k += nw) {
    const int q = NQ == 1 ? 0 : k & 1, gk = NQ == 1 ? k : k >> 1;
    const double* p = sums + (long)q * nsc;
    const int b = gk * 256 + lane;
    double v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = b + 32 * r < nsc ? ldv(&p[b + 32 * r]) : 0.0;
    double acc = v[0];
#pragma unroll
    for (int r = 1; r < 8; ++r) acc = acc + v[r];
    acc = warp_sum(acc);
    if (lane == 0) s_group[half][q][gk] = acc;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double acc = s_group[half][q][0];
    for (int k = 1; k < ng; ++k) acc = acc + s_group[half][q][k];
    out[q] = acc;
  }
  return true;
}

template <int NQ, typename State>
__device__ __forceinline__ bool resident_total(State& S, VGrid& g, DevStatus* st, double (&out)[NQ]) {
  total_post<NQ>(S, g);
  return total_wait<NQ>(S, g, st, out);
}

}  // namespace
}  // namespace mgpu
