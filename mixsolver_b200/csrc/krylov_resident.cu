// krylov_resident.cu -- the mixed form's solves for systems that fit in the
// SMs' shared memory: the pressure PCG (FP64 conjugate gradients with the FP32
// Chebyshev-Jacobi polynomial) and the momentum BiCGStab of krylov_poly.cuh,
// bit for bit the same numbers, with another division of the work.
//
// What bounds the streaming kernels (k_pcg_mixed) on such systems is neither
// HBM nor arithmetic: a Chebyshev pass of a few hundred thousand rows costs a
// grid barrier (every block's stores made visible, one counter, polls) plus
// two dependent trips to L2 per row, whatever the row count. Here
//   - a block owns a contiguous range of rows (whole super-chunks) for the
//     whole solve and keeps its rows of the FP32 matrix and 16-bit local
//     column numbers in shared memory and its part of the polynomial's vectors
//     in registers;
//   - between two passes only the values other blocks need move: each row's
//     new value goes to global memory in one 8-byte word together with the
//     number of its exchange, and a block reads the words its rows refer to
//     until they carry that number. The data is its own signal, so a pass has
//     no barrier and no fence (the words are written and read by relaxed
//     64-bit accesses, which are single-copy atomic). Only the sums
//     take a barrier (exchanged as words too, they were slower from about a
//     hundred blocks on, each polling every block's sums);
//   - the words a block needs are found in the prologue: the 32-row words its
//     columns touch, in the window [first row - bw, last row + bw], bw = the
//     largest |column - row|.
// The sums keep the layout-independent tree of krylov_poly.cuh.
//
// Measured on a B200, one PCG iteration at degree 24 (streaming kernel ->
// here): 6,400 rows 243 -> 27 us, 42,253 rows 99 -> 35 us, 82,944 rows (5
// entries) 93 -> 40 us, 524,288 rows 181 -> 116 us; a BiCGStab iteration 42,253
// rows 24 -> 11 us, 524,288 rows 46 -> 33 us. A pass of the 524,288 rows is
// 1.7 us of shared-memory reads (48 B of matrix and 7 gathers a row) and 1.9 us
// of exchange. Blocks of 512 threads two per SM and of 1024 (64 registers a
// thread) were 10-25 % slower, by their spills.

#include <algorithm>
#include <cmath>

#include "exchange.cuh"
#include "krylov_poly.cuh"

namespace mgpu {
extern int g_resident_sms;         // krylov.cu: the resident_sms tuning key
extern unsigned g_spin_limit;      // spin_limit
extern unsigned g_exchange_limit;  // exchange_spin_limit
namespace {

// Blocks of 256 threads, two per SM, or of 512, one per SM; 128 registers each.
constexpr int kResidentThreads = 512;
constexpr int kPairRows = 9 * kSuperRows;  // rows of a block of 256 threads, at most
constexpr int kHaloRegs = 4;   // halo words of a warp whose rows stay in registers
constexpr int kHaloBatch = 16; // halo words of a warp whose polls are in flight together, at most

// What a block keeps for the whole solve: its rows in shared memory (byte
// offsets into it) and the words it exchanges. The window starts at offset 0:
// R own values, then 32 per halo word.
template <int WC>
struct Resident {
  int n, R, start, end;  // rows of the system, of a block, this block's range
  int wb, nhw, nb;       // first row of the window, halo words, blocks
  int cp, cps;           // chunk sums (2 x cps doubles)
  int va;                // float4: entries 0..3
  int vb;                // 7: float4, entries 4..6 and the inverse diagonal; 5: float2, entry 4 and the inverse diagonal
  int ia;                // 7: uint4, window byte offsets of columns 0..6, 16 bits each; 5: uint2, of columns 0..3
  int ib;                // 5: unsigned short, of column 4
  int words;             // unsigned short: halo word k covers rows wb + 32 * word ...
  int nsc;
  unsigned seq, rseq;    // exchanges and sums so far
  u64* ll;               // exchange words (2 parities of n)
  double* sums;          // super-chunk sums (2 halves x 2 sums x nsc)
  int hpw;               // halo words per warp, rounded up
  WaitLimits waits;
  int hrow[kHaloRegs];   // the rows this lane polls for the warp's first halo words
};

// Shared memory of a block (bytes); nhw halo words, window of wwin words.
__host__ __device__ inline int resident_win_bytes(int R, int nhw, int wwin) {
  const int win = 4 * R + 128 * (nhw + 1), scratch = 4 * wwin;  // the prologue's word ranks, in the window's place
  return ((win > scratch ? win : scratch) + 15) & ~15;
}
__host__ __device__ inline int resident_window_words(int R, int bw) { return R / 32 + 2 * ((bw + 31) / 32); }
// matrix planes: values, then window offsets and the halo word list (its last
// entry: their number, in a page)
__host__ __device__ inline int resident_values(int WC, int R) { return (WC == 7 ? 32 : 24) * R; }
__host__ __device__ inline int resident_places(int WC, int R, int nhw) {
  return (WC == 7 ? 16 : 10) * R + ((2 * nhw + 2 + 15) & ~15);
}
// a page in global memory, whole lines
__host__ __device__ inline int page_bytes(int WC, int R, int nhw) {
  return (resident_values(WC, R) + resident_places(WC, R, nhw) + 127) & ~127;
}
__host__ __device__ inline int resident_smem(int WC, int R, int bw, int nhw, int cps) {
  return resident_win_bytes(R, nhw, resident_window_words(R, bw)) + 16 * cps + resident_values(WC, R) + resident_places(WC, R, nhw);
}

template <int WC>
__device__ __forceinline__ void resident_views(Resident<WC>& m, int R, int bw, int nhw, int cps) {
  m.cp = resident_win_bytes(R, nhw, resident_window_words(R, bw));
  m.cps = cps;
  m.va = m.cp + 16 * cps;
  m.vb = m.va + 16 * R;
  m.ia = m.vb + (WC == 7 ? 16 : 8) * R;
  m.ib = m.ia + (WC == 7 ? 16 : 8) * R;
  m.words = m.ib + (WC == 7 ? 0 : 2) * R;
}

__device__ __forceinline__ float win_at(unsigned off) {
  return *reinterpret_cast<const float*>(block_smem + off);
}

// f(entry, byte offset of its column in the window) over the row's entries
template <int WC, typename F>
__device__ __forceinline__ void resident_cols(const Resident<WC>& m, int l, F&& f) {
  if constexpr (WC == 7) {
    const uint4 c = smem_at<uint4>(m.ia, l);
    f(0, c.x & 0xffffu);
    f(1, c.x >> 16);
    f(2, c.y & 0xffffu);
    f(3, c.y >> 16);
    f(4, c.z & 0xffffu);
    f(5, c.z >> 16);
    f(6, c.w);
  } else {
    const uint2 c = smem_at<uint2>(m.ia, l);
    f(0, c.x & 0xffffu);
    f(1, c.x >> 16);
    f(2, c.y & 0xffffu);
    f(3, c.y >> 16);
    f(4, (unsigned)smem_at<unsigned short>(m.ib, l));
  }
}

// One row of the FP32 product: entries in ELL order as in spmv32_rows (entries
// past the row's width are value 0 at the row itself).
template <int WC>
__device__ __forceinline__ float resident_row(const Resident<WC>& m, int l, float& dinv) {
  float v[WC];
  const float4 a = smem_at<float4>(m.va, l);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = a.z;
  v[3] = a.w;
  if constexpr (WC == 7) {
    const float4 b = smem_at<float4>(m.vb, l);
    v[4] = b.x;
    v[5] = b.y;
    v[6] = b.z;
    dinv = b.w;
  } else {
    const float2 b = smem_at<float2>(m.vb, l);
    v[4] = b.x;
    dinv = b.y;
  }
  float acc = 0.0f;
  resident_cols<WC>(m, l, [&](int t, unsigned off) { acc = fmaf(v[t], win_at(off), acc); });
  return acc;
}

// The row's inverse diagonal.
template <int WC>
__device__ __forceinline__ float resident_dinv(const Resident<WC>& m, int l) {
  if constexpr (WC == 7)
    return smem_at<float4>(m.vb, l).w;
  else
    return smem_at<float2>(m.vb, l).y;
}

// The rows row[0 .. HB) of this lane, polled until they carry number seq, into
// the window from halo word w0 in steps of the block's warps. Straight-line: a
// taken branch a word costs more than the word (nhw = 6 words with 16 guarded
// polls: 1.09 us an exchange, with 8: 0.74 us); words and lanes past the halo
// poll a row of this block instead and land in the window's spare word.
template <int HB, int WC>
__device__ __forceinline__ bool halo_fetch(const Resident<WC>& S, const u64* llb, unsigned seq,
                                           const int* row, int w0, DevStatus* st) {
  const int T = blockDim.x, lane = threadIdx.x & 31, nw = T >> 5;
  u64 v[HB];
#pragma unroll
  for (int q = 0; q < HB; ++q) v[q] = ld_word(llb + row[q]);
  unsigned left = S.waits.value;
  while (true) {
    unsigned bad = 0u;
#pragma unroll
    for (int q = 0; q < HB; ++q) bad |= (unsigned)(v[q] >> 32) ^ seq;
    if (bad == 0u) break;
    if (!keep_polling(left, st)) return false;
#pragma unroll
    for (int q = 0; q < HB; ++q)
      if ((unsigned)(v[q] >> 32) != seq) v[q] = ld_word(llb + row[q]);
  }
#pragma unroll
  for (int q = 0; q < HB; ++q)
    smem_at<float>(0, S.R + 32 * min(w0 + q * nw, S.nhw) + lane) = __uint_as_float((unsigned)v[q]);
  return true;
}

// The row lane polls for halo word w.
template <int WC>
__device__ __forceinline__ int halo_row(const Resident<WC>& S, int w) {
  const int lane = threadIdx.x & 31;
  const int own = min(S.start + lane, S.end - 1);
  const int row = w < S.nhw ? S.wb + 32 * (int)smem_at<unsigned short>(S.words, w) + lane : own;
  return row < S.n ? row : own;
}

// An exchange, number seq. Publish: this block's new values z (registers) to
// its words. Receive: they go to its own window too, and the halo words are
// read until they carry the number; the closing barrier also ends the reads of
// the window before. Words of the other parity may still be read by a slower
// neighbour; these are free: a block publishes exchange s + 2 only after it has
// read the words s + 1 of every block it exchanges with (the pattern is
// symmetric), which those published after reading all of their words s.
// receive returns false when a bounded poll ran out.
template <int WC, int K>
__device__ __forceinline__ void resident_publish(const Resident<WC>& S, const float (&z)[K], unsigned seq) {
  u64* llb = S.ll + (long)(seq & 1u) * S.n;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = S.start + k * (int)blockDim.x + (int)threadIdx.x;
    if (i < S.end) st_word(llb + i, pack_word(__float_as_uint(z[k]), seq));
  }
}

template <int WC, int K>
__device__ __forceinline__ bool resident_receive(const Resident<WC>& S, const float (&z)[K], unsigned seq,
                                                 DevStatus* st) {
  const int T = blockDim.x, tid = threadIdx.x, warp = tid >> 5, nw = T >> 5;
  const u64* llb = S.ll + (long)(seq & 1u) * S.n;
  __syncthreads();  // the pass's reads of the window are done
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int l = k * T + tid;
    if (l < S.R) smem_at<float>(0, l) = z[k];
  }
  // the polls start only now: sent right after the stores, the first ones come
  // back before the neighbours' words
  bool ok = true;
  if (S.hpw > 0) {
    if (S.hpw <= 1)
      ok = halo_fetch<1>(S, llb, seq, S.hrow, warp, st);
    else if (S.hpw <= 2)
      ok = halo_fetch<2>(S, llb, seq, S.hrow, warp, st);
    else if (S.hpw <= 4)
      ok = halo_fetch<4>(S, llb, seq, S.hrow, warp, st);
    else
      for (int w0 = warp; w0 < S.nhw && ok; w0 += kHaloBatch * nw) {
        int row[kHaloBatch];
        if (w0 + 8 * nw >= S.nhw) {
#pragma unroll
          for (int q = 0; q < 8; ++q) row[q] = halo_row(S, w0 + q * nw);
          ok = halo_fetch<8>(S, llb, seq, row, w0, st);
        } else {
#pragma unroll
          for (int q = 0; q < kHaloBatch; ++q) row[q] = halo_row(S, w0 + q * nw);
          ok = halo_fetch<kHaloBatch>(S, llb, seq, row, w0, st);
        }
      }
  }
  return __syncthreads_and(ok) != 0;
}

// The block's next exchange; between() runs while the words travel.
template <int WC, int K, typename F>
__device__ __forceinline__ bool resident_exchange(Resident<WC>& S, const float (&z)[K], DevStatus* st, F&& between) {
  const unsigned seq = ++S.seq;
  if (S.nb > 1) resident_publish<WC, K>(S, z, seq);
  between();
  return resident_receive<WC, K>(S, z, seq, st);
}

// The rows of the block's range into shared memory: the window's halo words,
// ranked in ascending order, the window offsets of the columns, the FP32 values
// and inverse diagonals; the FP64 ELL values (PCG); the exchange words cleared;
// the chunk sums of b.b and of the zero diagonals.
template <int WC, int K, bool PCG>
__device__ __forceinline__ void resident_build(const KrylovArgs& a, const MixedArgs& m, Resident<WC>& S) {
  const int T = blockDim.x, tid = threadIdx.x, s0 = S.start, e0 = s0 + S.R;
  const int lane = tid & 31, warp = tid >> 5, nw = T >> 5;
  const int W = m.ell_w, ld = m.ell_ld;
  S.wb = max(0, s0 - (m.plan.bw + 31) / 32 * 32);
  const int nwords = (min(S.n, e0 + m.plan.bw) - S.wb + 31) / 32;
  unsigned* rank_of = reinterpret_cast<unsigned*>(block_smem);
  __shared__ unsigned s_warp[32];
  __shared__ unsigned s_run;
  for (int w = tid; w < nwords; w += T) rank_of[w] = 0u;
  if (tid == 0) s_run = 0u;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = s0 + k * T + tid;
    if (i < S.end)
#pragma unroll
      for (int t = 0; t < WC; ++t)
        if (t < W) {
          const int c = m.ell_col[t * ld + i];
          if (c < s0 || c >= e0) rank_of[(c - S.wb) >> 5] = 1u;  // every writer stores the same value
        }
  }
  __syncthreads();
  for (int w0 = 0; w0 < nwords; w0 += T) {
    const int w = w0 + tid;
    const bool on = w < nwords && rank_of[w] != 0u;
    const unsigned bal = __ballot_sync(0xffffffffu, on);
    if (lane == 0) s_warp[warp] = __popc(bal);
    __syncthreads();
    unsigned before = s_run;
    for (int q = 0; q < warp; ++q) before += s_warp[q];
    const unsigned rank = before + __popc(bal & ((1u << lane) - 1u));
    __syncthreads();
    if (tid == T - 1) s_run = before + __popc(bal);
    if (on) {
      rank_of[w] = rank;
      smem_at<unsigned short>(S.words, (int)rank) = (unsigned short)w;
    }
    __syncthreads();
  }
  S.nhw = (int)s_run;
  S.hpw = (S.nhw + nw - 1) / nw;
#pragma unroll
  for (int q = 0; q < kHaloRegs; ++q) S.hrow[q] = halo_row(S, warp + q * nw);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int l = k * T + tid, i = s0 + l;
    double c[2] = {0.0, 0.0};
    float v[WC];
    unsigned lc[WC];
    float dv = 0.0f;
#pragma unroll
    for (int t = 0; t < WC; ++t) {
      v[t] = 0.0f;
      lc[t] = 4u * (unsigned)l;
    }
    if (i < S.end) {
      const int rb = a.row_ptr[i], nr = a.row_ptr[i + 1] - rb;
#pragma unroll
      for (int t = 0; t < WC; ++t)
        if (t < W) {
          const double av = t < nr ? a.aval[rb + t] : 0.0;
          v[t] = (float)av;
          if (PCG) m.ell64[t * ld + i] = av;  // q = A p
          const int cc = m.ell_col[t * ld + i];
          lc[t] = 4u * (cc >= s0 && cc < e0
                            ? (unsigned)(cc - s0)
                            : (unsigned)S.R + 32u * rank_of[(cc - S.wb) >> 5] + (unsigned)((cc - S.wb) & 31));
        }
      if (a.zero_x) a.x[i] = 0.0;
      const double dg = a.aval[a.diag[i]];
      if (fabs(dg) < DTINY) c[1] = 1.0;
      dv = (float)(1.0 / dg);
      c[0] = a.b[i] * a.b[i];
      S.ll[i] = 0ull;
      S.ll[(long)S.n + i] = 0ull;
    }
    if (l < S.R) {
      smem_at<float4>(S.va, l) = make_float4(v[0], v[1], v[2], v[3]);
      if constexpr (WC == 7) {
        smem_at<float4>(S.vb, l) = make_float4(v[4], v[5], v[6], dv);
        smem_at<uint4>(S.ia, l) = make_uint4(lc[0] | lc[1] << 16, lc[2] | lc[3] << 16, lc[4] | lc[5] << 16, lc[6]);
      } else {
        smem_at<float2>(S.vb, l) = make_float2(v[4], dv);
        smem_at<uint2>(S.ia, l) = make_uint2(lc[0] | lc[1] << 16, lc[2] | lc[3] << 16);
        smem_at<unsigned short>(S.ib, l) = (unsigned short)lc[4];
      }
    }
    resident_put<2>(S.cp, S.cps, k, c);
  }
}

// The block's rows, then b.b and the count of zero diagonals; the barrier puts
// every block's cleared words before the first exchange.
template <int WC, int K, bool PCG>
__device__ __forceinline__ bool resident_prologue(const KrylovArgs& a, const MixedArgs& m, VGrid& g, Resident<WC>& S,
                                                  double& bnrm, bool& diag_bad) {
  resident_build<WC, K, PCG>(a, m, S);
  if (!vg_sync(g, a.st)) return false;
  double v[2];
  if (!resident_total<2>(S, g, a.st, v)) return false;
  bnrm = sqrt(v[0]);
  diag_bad = v[1] != 0.0;
  return true;
}

__shared__ float2 s_cheb[64];  // the polynomial's recurrence coefficients

// cheb_apply's coefficients on [lmax / ratio, lmax] into s_cheb (every thread
// calls it); returns 1 / theta of the first term.
__device__ __forceinline__ float cheb_table(double lmax, double ratio, int degree) {
  const double lmin = lmax / ratio;
  const double th = 0.5 * (lmax + lmin), de = 0.5 * (lmax - lmin), sg = th / de;
  if (threadIdx.x == 0) {
    double rho0 = 1.0 / sg;
    for (int j = 1; j < degree; ++j) {
      const double rho1 = 1.0 / (2.0 * sg - rho0);
      s_cheb[j] = make_float2((float)(rho1 * rho0), (float)(2.0 * rho1 / de));
      rho0 = rho1;
    }
  }
  __syncthreads();
  return (float)(1.0 / th);
}

// The Chebyshev-Jacobi polynomial of cheb_apply on the block's rows: on entry
// z holds z0 (registers, exchanged); on return z is the result, exchanged, and
// rz the sum r64.z.
template <int WC, int K>
__device__ __forceinline__ bool resident_cheb(Resident<WC>& S, VGrid& g, DevStatus* st, int degree, const float (&rr)[K],
                                              float (&z)[K], const double* r64, double& rz) {
  const int T = blockDim.x, tid = threadIdx.x;
  float d[K];
#pragma unroll
  for (int k = 0; k < K; ++k) d[k] = z[k];
  for (int j = 1; j < degree; ++j) {
    const float2 c = s_cheb[j];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int l = k * T + tid;
      if (l < S.R) {
        float dinv;
        const float az = resident_row<WC>(S, l, dinv);
        const float res = dinv * (rr[k] - az);
        d[k] = fmaf(c.x, d[k], c.y * res);
        z[k] = z[k] + d[k];
      }
    }
    if (j == degree - 1) break;
    if (!resident_exchange<WC, K>(S, z, st, [] {})) return false;
  }
  // the result and its sum travel together
  if (!resident_exchange<WC, K>(S, z, st, [&] {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int i = S.start + k * T + tid;
          const double c[1] = {i < S.end ? r64[i] * (double)z[k] : 0.0};
          resident_put<1>(S.cp, S.cps, k, c);
        }
        total_post<1>(S, g);
      }))
    return false;
  double t[1];
  if (!total_wait<1>(S, g, st, t)) return false;
  rz = t[0];
  return true;
}

// pcg_hybrid (krylov_poly.cuh) on resident rows: the same recurrences, sums
// and decisions.
template <int WC, int K>
__device__ __forceinline__ void resident_pcg(const KrylovArgs& a, const MixedArgs& m, VGrid& g, Resident<WC>& S, double bnrm,
                             double rnorm0, float inv_th) {
  const int T = blockDim.x, tid = threadIdx.x, ld = m.ell_ld, W = m.ell_w;
  double *rs = a.r, *p = a.p, *pn = a.s;  // the direction is double-buffered
  const double* __restrict__ ev = m.ell64;
  const double sc = 1.0 / rnorm0;
  const double stop = a.tol * bnrm * sc;
  const double stop2 = stop * stop;
  float z[K], rr[K];
  double pk[K], qk[K];
  // row i of the scaled residual: its FP32 copy and the first Chebyshev term
  auto begin_row = [&](int k, int i, double ri) {
    rs[i] = ri;
    rr[k] = (float)ri;
    z[k] = resident_dinv<WC>(S, k * T + tid) * rr[k] * inv_th;
  };
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = S.start + k * T + tid;
    z[k] = rr[k] = 0.0f;
    if (i < S.end) begin_row(k, i, ldv(&a.r[i]) * sc);
  }
  if (!resident_exchange<WC, K>(S, z, a.st, [] {})) return;
  double rz = 0.0, rnorm = rnorm0;
  int total = 0, ierr = 0;
  bool first = true;
  while (true) {
    double rzn;
    if (!resident_cheb<WC, K>(S, g, a.st, m.cheb_k, rr, z, rs, rzn)) return;
    double beta = 0.0;
    if (!first) {
      if (fabs(rz) < DTINY) {
        ierr = 2;
        break;
      }
      beta = rzn / rz;
    }
    rz = rzn;
    ++total;
    // pn := z + beta p, q := A pn: z from the window, p of the rows' columns
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int l = k * T + tid, i = S.start + l;
      double c[1] = {0.0};
      pk[k] = qk[k] = 0.0;
      if (i < S.end) {
        double v[WC], x[WC];
        resident_cols<WC>(S, l, [&](int t, unsigned off) {
          v[t] = t < W ? ev[t * ld + i] : 0.0;
          const int lc = (int)(off >> 2);
          const int col = lc < S.R ? S.start + lc : S.wb + 32 * (int)smem_at<unsigned short>(S.words, (lc - S.R) >> 5) + (lc & 31);
          x[t] = first ? 0.0 : ldv(&p[col]);
        });
        resident_cols<WC>(S, l, [&](int t, unsigned off) {
          const double zt = (double)win_at(off);
          x[t] = first ? zt : fma(beta, x[t], zt);
        });
        double acc = 0.0;
#pragma unroll
        for (int t = 0; t < WC; ++t)
          if (t < W) acc = fma(v[t], x[t], acc);
        const double pi = first ? (double)z[k] : fma(beta, p[i], (double)z[k]);
        pn[i] = pi;
        pk[k] = pi;
        qk[k] = acc;
        c[0] = pi * acc;
      }
      resident_put<1>(S.cp, S.cps, k, c);
    }
    {
      double* t = p;
      p = pn;
      pn = t;
    }
    first = false;
    double pq[1];
    if (!resident_total<1>(S, g, a.st, pq)) return;  // the direction is gathered next iteration
    if (fabs(pq[0]) < DTINY) {
      ierr = 2;
      break;
    }
    const double al = rz / pq[0];
    const double ax = al * rnorm0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = S.start + k * T + tid;
      double c[1] = {0.0};
      if (i < S.end) {
        const double ri = fma(-al, qk[k], rs[i]);
        begin_row(k, i, ri);
        c[0] = ri * ri;
      }
      resident_put<1>(S.cp, S.cps, k, c);
    }
    if (!resident_exchange<WC, K>(S, z, a.st, [&] {
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int i = S.start + k * T + tid;
            if (i < S.end) a.x[i] = fma(ax, pk[k], a.x[i]);
          }
          total_post<1>(S, g);
        }))
      return;
    double s2[1];
    if (!total_wait<1>(S, g, a.st, s2)) return;
    if (!(s2[0] <= stop2 || total >= a.maxit)) continue;
    // r = b - A x in FP64 decides (the sum's barrier shows every block's x)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = S.start + k * T + tid;
      double c[1] = {0.0};
      if (i < S.end) {
        const double ri = a.b[i] - row_spmv64<false>(a, a.x, i);
        begin_row(k, i, ri * sc);
        c[0] = ri * ri;
      }
      resident_put<1>(S.cp, S.cps, k, c);
    }
    if (!resident_exchange<WC, K>(S, z, a.st, [] {})) return;
    double t2[1];
    if (!resident_total<1>(S, g, a.st, t2)) return;  // x is written again only after every block has read it
    rnorm = sqrt(t2[0]);
    const double res = rnorm / bnrm;
    if (res <= a.tol) {
      write_result_m(a, g, total, res, 0);
      return;
    }
    if (total >= a.maxit) {
      ierr = 1;
      break;
    }
    first = true;  // the recursive residual had drifted: restart from the true one
  }
  write_result_m(a, g, total, rnorm / bnrm, ierr);
}

// The block's part of the system: its range, its views and the prologue. False
// when the kernel must leave (a wait ran out, or the result is already known:
// b = 0, or a zero diagonal with code diag_code).
template <int WC, int K, bool PCG>
__device__ __forceinline__ bool resident_begin(const KrylovArgs& a, const MixedArgs& m, VGrid& g, Resident<WC>& S,
                                               WaitLimits waits, int R, int nhw_max, int diag_code, double& bnrm) {
  const int n = a.n;
  S.waits = waits;
  S.n = n;
  S.R = R;
  S.nb = g.nb;
  S.start = g.rank * R;
  S.end = min(n, S.start + R);
  S.nsc = (n + kSuperRows - 1) / kSuperRows;
  S.seq = S.rseq = 0u;
  S.sums = m.red;
  S.ll = reinterpret_cast<u64*>(m.w32);  // the FP32 work vectors' space
  resident_views<WC>(S, R, m.plan.bw, nhw_max, K * (blockDim.x / 32));
  bool diag_bad;
  if (!resident_prologue<WC, K, PCG>(a, m, g, S, bnrm, diag_bad)) return false;
  if (bnrm == 0.0) {
    for (int i = S.start + threadIdx.x; i < S.end; i += blockDim.x) a.x[i] = 0.0;
    write_result_m(a, g, 0, 0.0, 0);
    return false;
  }
  if (diag_bad) {
    write_result_m(a, g, 0, 0.0, diag_code);
    return false;
  }
  return true;
}

// nhw_max: the halo words the shared memory was sized for.
template <int WC, int K>
__global__ void __launch_bounds__(kResidentThreads, 1) k_pcg_resident(KrylovArgs a, MixedArgs m, WaitLimits waits,
                                                                       int R, int nhw_max) {
  if (a.st->abort) return;
  VGrid g = whole_grid(a.bar, a.partials, true);
  const int T = blockDim.x, tid = threadIdx.x;
  Resident<WC> S;
  double bnrm;
  if (!resident_begin<WC, K, true>(a, m, g, S, waits, R, nhw_max, 2, bnrm)) return;
  // Gershgorin bound of D^-1 A (a maximum is exact in any order), b - A x
  double gm = 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = S.start + k * T + tid;
    double c[1] = {0.0};
    if (i < S.end) {
      double s = 0.0;
      for (int q = a.row_ptr[i]; q < a.row_ptr[i + 1]; ++q) s += fabs(a.aval[q]);
      gm = fmax(gm, s / fabs(a.aval[a.diag[i]]));
      const double ri = a.b[i] - row_spmv64<false>(a, a.x, i);
      a.r[i] = ri;
      c[0] = ri * ri;
    }
    resident_put<1>(S.cp, S.cps, k, c);
  }
  if (!vg_max<false>(gm, g, a.st)) return;  // its barrier: nobody reads x any more
  double rn[1];
  if (!resident_total<1>(S, g, a.st, rn)) return;
  const double rnorm = sqrt(rn[0]);
  const double res = rnorm / bnrm;
  if (res <= a.tol) {
    write_result_m(a, g, 0, res, 0);
    return;
  }
  const float inv_th = cheb_table(gm, m.cheb_ratio, m.cheb_k);
  resident_pcg<WC, K>(a, m, g, S, bnrm, rnorm, inv_th);
}

// ---------------------------------------------------------------------------
// Larger systems: the blocks' rows in turns
// ---------------------------------------------------------------------------

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// The PCG of resident_pcg for a system larger than the SMs' shared memory. What
// bounds it when streamed (k_pcg_mixed) is the matrix: every Chebyshev pass
// reads all of it, 40 or 56 bytes a row, from HBM. Here the rows are cut into
// pages (what a resident block holds: planes of matrix rows, window offsets and
// halo words, built once a solve in global memory). Block b takes pages b, b +
// nb, ... in turn, loads one into shared memory and runs plan.steps polynomial
// steps on it before the next, exchanging values step by step with the blocks
// that hold the neighbouring pages, so the matrix is read once per plan.steps
// passes. There is no barrier: page p's step s waits for the words of step
// s - 1 of the pages its rows refer to, at most r = ceil(bw / rows) pages
// ahead. No wait is circular: within a sweep over the pages, order the steps
// by (p + s r); a step waits for words of lesser or equal rank and lesser s,
// and a block's turn at page p + nb starts after its last step at p, of rank
// p + steps r < p + nb + r while (steps - 1) r < nb (the plan keeps to half of
// that); a sweep never waits for a later one. The other vectors stream.
// Measured on a B200, an iteration at degree 48 streamed -> here: 2,000,376 rows of
// 7 entries 1,541 -> 1,234 to 1,315 us, 2,500,000 rows of 5 (a grid) 1,569 -> 974 to
// 1,074 us (more sizes at turns_pay). A step of a page takes 1.7 us of shared-memory reads and 2.9 us of
// exchange (1.9 in the resident solve: here L2 also carries the pages), a turn 4.8 us
// to load.
template <int WC, int K>
__global__ void __launch_bounds__(256, 2) k_pcg_paged(KrylovArgs a, MixedArgs m, WaitLimits waits) {
  if (a.st->abort) return;
  VGrid g = whole_grid(a.bar, a.partials, true);
  const int n = a.n, T = blockDim.x, tid = threadIdx.x, R = m.plan.rows, W = m.ell_w, ld = m.ell_ld;
  const int npages = (n + R - 1) / R, degree = m.cheb_k;
  const int vbytes = resident_values(WC, R), pb = vbytes + resident_places(WC, R, m.plan.words);
  const long pstep = page_bytes(WC, R, m.plan.words);
  const int warp = tid >> 5, nw = T >> 5;
  Resident<WC> S;
  S.waits = waits;
  S.n = n;
  S.R = R;
  S.nb = npages;
  S.nsc = (n + kSuperRows - 1) / kSuperRows;
  S.seq = S.rseq = 0u;
  S.sums = m.red;
  S.ll = reinterpret_cast<u64*>(m.w32);
  float *dch = m.w32 + 4l * n, *rr = m.w32 + 5l * n, *zf = m.w32 + 6l * n;
  resident_views<WC>(S, R, m.plan.bw, m.plan.words, K * (T / 32));
  // the pages follow the FP32 CSR values
  unsigned char* const pages = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<unsigned long long>(m.a32 + a.row_ptr[n]) + 127) & ~127ull);
  auto turn = [&](int p) {
    S.start = p * R;
    S.end = min(n, S.start + R);
    S.wb = max(0, S.start - (m.plan.bw + 31) / 32 * 32);
  };
// a page's rows, in tiles of T
#define MGPU_PAGE_ROWS(k, i) \
  for (int k = 0; k < K; ++k) \
    if (const int i = S.start + k * T + tid; true)
  // the pages, b.b, the zero diagonals
  double gm = 0.0;
  ++S.rseq;
  for (int p = g.rank; p < npages; p += g.nb) {
    turn(p);
    __syncthreads();  // the page before has left shared memory
    resident_build<WC, K, true>(a, m, S);
    if (tid == 0) smem_at<unsigned short>(S.words, m.plan.words) = (unsigned short)S.nhw;
    MGPU_PAGE_ROWS(k, i) {
      if (i < S.end) {
        m.dinv[i] = resident_dinv<WC>(S, k * T + tid);
        double s = 0.0;
        for (int q = a.row_ptr[i]; q < a.row_ptr[i + 1]; ++q) s += fabs(a.aval[q]);
        gm = fmax(gm, s / fabs(a.aval[a.diag[i]]));
      }
    }
    super_sums<2>(S);
    uint4* page = reinterpret_cast<uint4*>(pages + p * pstep);
    for (int o = tid; o < pb / 16; o += T) page[o] = smem_at<uint4>(S.va, o);
  }
  vg_arrive(g);
  double v2[2];
  if (!total_wait<2>(S, g, a.st, v2)) return;
  const double bnrm = sqrt(v2[0]);
  if (bnrm == 0.0) {
    for (int p = g.rank; p < npages; p += g.nb) {
      turn(p);
      MGPU_PAGE_ROWS(k, i) {
        if (i < S.end) a.x[i] = 0.0;
      }
    }
    write_result_m(a, g, 0, 0.0, 0);
    return;
  }
  if (v2[1] != 0.0) {
    write_result_m(a, g, 0, 0.0, 2);
    return;
  }
  // r = b - A x
  ++S.rseq;
  for (int p = g.rank; p < npages; p += g.nb) {
    turn(p);
    __syncthreads();
    MGPU_PAGE_ROWS(k, i) {
      double c[1] = {0.0};
      if (i < S.end) {
        const double ri = a.b[i] - row_spmv64<false>(a, a.x, i);
        a.r[i] = ri;
        c[0] = ri * ri;
      }
      resident_put<1>(S.cp, S.cps, k, c);
    }
    super_sums<1>(S);
  }
  if (!vg_max<false>(gm, g, a.st)) return;
  vg_arrive(g);
  double t1[1];
  if (!total_wait<1>(S, g, a.st, t1)) return;
  const double rnorm0 = sqrt(t1[0]);
  double res = rnorm0 / bnrm, rnorm = rnorm0;
  if (res <= a.tol) {
    write_result_m(a, g, 0, res, 0);
    return;
  }
  const float inv_th = cheb_table(gm, m.cheb_ratio, degree);
  double *rs = a.r, *pd = a.p, *pn = a.s, *qd = a.v;
  const double* __restrict__ ev = m.ell64;
  const int* __restrict__ ecol = m.ell_col;
  const float* __restrict__ dinv = m.dinv;
  const double sc = 1.0 / rnorm0, stop = a.tol * bnrm * sc, stop2 = stop * stop;
  // row i of the scaled residual: its FP32 copy, the first Chebyshev term, which
  // is published as exchange S.seq
  auto begin_row = [&](int i, double ri) {
    rs[i] = ri;
    const float rf = (float)ri;
    rr[i] = rf;
    const float z0 = dinv[i] * rf * inv_th;
    dch[i] = z0;
    st_word(S.ll + (long)(S.seq & 1u) * n + i, pack_word(__float_as_uint(z0), S.seq));
  };
  ++S.seq;
  for (int p = g.rank; p < npages; p += g.nb) {
    turn(p);
    MGPU_PAGE_ROWS(k, i) {
      if (i < S.end) begin_row(i, a.r[i] * sc);
    }
  }
  double rz = 0.0;
  int total = 0, ierr = 0;
  bool first = true;
  while (true) {
    // the polynomial: sweeps of up to plan.steps steps a page
    ++S.rseq;
    for (int done = 0; done < degree - 1;) {
      const int ns = min(m.plan.steps, degree - 1 - done);
      const bool final = done + ns == degree - 1;
      for (int p = g.rank; p < npages; p += g.nb) {
        turn(p);
        __syncthreads();  // the page before has left shared memory
        const unsigned char* page = pages + p * pstep;
        for (int o = 16 * tid; o < pb; o += 16 * T) cp_async16(block_smem + S.va + o, page + o);
        float z[K], d[K], rv[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int i = S.start + k * T + tid;
          z[k] = d[k] = rv[k] = 0.0f;
          if (i < S.end) {
            z[k] = __uint_as_float((unsigned)ld_word(S.ll + (long)(S.seq & 1u) * n + i));
            d[k] = dch[i];
            rv[k] = rr[i];
          }
        }
        // the block's next page on its way to L2 while this one is at work
        {
          const int pnext = p + g.nb < npages ? p + g.nb : g.rank;
          const unsigned char* next = pages + pnext * pstep;
          for (int o = 128 * tid; o < pb; o += 128 * T) prefetch_l2(next + o);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        S.nhw = smem_at<unsigned short>(S.words, m.plan.words);
        S.hpw = (S.nhw + nw - 1) / nw;
#pragma unroll
        for (int q = 0; q < kHaloRegs; ++q) S.hrow[q] = halo_row(S, warp + q * nw);
        for (int j = 1; j <= ns; ++j) {
          if (!resident_receive<WC, K>(S, z, S.seq + j - 1, a.st)) return;
          const float2 c = s_cheb[done + j];
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int l = k * T + tid;
            if (l < R) {
              float di;
              const float az = resident_row<WC>(S, l, di);
              const float rk = di * (rv[k] - az);
              d[k] = fmaf(c.x, d[k], c.y * rk);
              z[k] = z[k] + d[k];
            }
          }
          resident_publish<WC, K>(S, z, S.seq + j);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int i = S.start + k * T + tid;
          double c[1] = {0.0};
          if (i < S.end) {
            if (final) {
              zf[i] = z[k];
              c[0] = rs[i] * (double)z[k];
            } else {
              dch[i] = d[k];
            }
          }
          if (final) resident_put<1>(S.cp, S.cps, k, c);
        }
        if (final) super_sums<1>(S);
      }
      S.seq += ns;
      done += ns;
    }
    vg_arrive(g);
    if (!total_wait<1>(S, g, a.st, t1)) return;
    const double rzn = t1[0];
    double beta = 0.0;
    if (!first) {
      if (fabs(rz) < DTINY) {
        ierr = 2;
        break;
      }
      beta = rzn / rz;
    }
    rz = rzn;
    ++total;
    // pn := z + beta p, q := A pn
    ++S.rseq;
    for (int p = g.rank; p < npages; p += g.nb) {
      turn(p);
      __syncthreads();
#pragma unroll 2
      MGPU_PAGE_ROWS(k, i) {
        double c[1] = {0.0};
        if (i < S.end) {
          double v[WC], x[WC];
          int cc[WC];
#pragma unroll
          for (int t = 0; t < WC; ++t)
            if (t < W) {
              cc[t] = ecol[t * ld + i];
              v[t] = ev[t * ld + i];
            }
#pragma unroll
          for (int t = 0; t < WC; ++t)
            if (t < W) x[t] = first ? (double)ldv(&zf[cc[t]]) : fma(beta, ldv(&pd[cc[t]]), (double)ldv(&zf[cc[t]]));
          double acc = 0.0;
#pragma unroll
          for (int t = 0; t < WC; ++t)
            if (t < W) acc = fma(v[t], x[t], acc);
          const double pi = first ? (double)zf[i] : fma(beta, pd[i], (double)zf[i]);
          pn[i] = pi;
          qd[i] = acc;
          c[0] = pi * acc;
        }
        resident_put<1>(S.cp, S.cps, k, c);
      }
      super_sums<1>(S);
    }
    {
      double* t = pd;
      pd = pn;
      pn = t;
    }
    first = false;
    vg_arrive(g);
    if (!total_wait<1>(S, g, a.st, t1)) return;
    if (fabs(t1[0]) < DTINY) {
      ierr = 2;
      break;
    }
    const double al = rz / t1[0];
    const double ax = al * rnorm0;
    ++S.rseq;
    ++S.seq;
    for (int p = g.rank; p < npages; p += g.nb) {
      turn(p);
      __syncthreads();
#pragma unroll 2
      MGPU_PAGE_ROWS(k, i) {
        double c[1] = {0.0};
        if (i < S.end) {
          a.x[i] = fma(ax, pd[i], a.x[i]);
          const double ri = fma(-al, qd[i], rs[i]);
          begin_row(i, ri);
          c[0] = ri * ri;
        }
        resident_put<1>(S.cp, S.cps, k, c);
      }
      super_sums<1>(S);
    }
    vg_arrive(g);
    if (!total_wait<1>(S, g, a.st, t1)) return;
    if (!(t1[0] <= stop2 || total >= a.maxit)) continue;
    // r = b - A x in FP64 decides
    ++S.rseq;
    ++S.seq;
    for (int p = g.rank; p < npages; p += g.nb) {
      turn(p);
      __syncthreads();
      MGPU_PAGE_ROWS(k, i) {
        double c[1] = {0.0};
        if (i < S.end) {
          const double ri = a.b[i] - row_spmv64<false>(a, a.x, i);
          begin_row(i, ri * sc);
          c[0] = ri * ri;
        }
        resident_put<1>(S.cp, S.cps, k, c);
      }
      super_sums<1>(S);
    }
    vg_arrive(g);
    if (!total_wait<1>(S, g, a.st, t1)) return;
    rnorm = sqrt(t1[0]);
    res = rnorm / bnrm;
    if (res <= a.tol) {
      write_result_m(a, g, total, res, 0);
      return;
    }
    if (total >= a.maxit) {
      ierr = 1;
      break;
    }
    first = true;
  }
  write_result_m(a, g, total, rnorm / bnrm, ierr);
}
#undef MGPU_PAGE_ROWS

// bicgstab_mixed_body (krylov_poly.cuh) on resident rows: the FP32 vectors in
// registers, one exchange for each of the two products, the same recurrences,
// sums and decisions.
template <int WC, int K>
__global__ void __launch_bounds__(kResidentThreads, 1) k_bicgstab_resident(KrylovArgs a, MixedArgs m, WaitLimits waits,
                                                                            int R, int nhw_max) {
  if (a.st->abort) return;
  VGrid g = whole_grid(a.bar, a.partials, true);
  const int T = blockDim.x, tid = threadIdx.x;
  Resident<WC> S;
  double bnrm;
  if (!resident_begin<WC, K, false>(a, m, g, S, waits, R, nhw_max, 12, bnrm)) return;
  float r[K], r0[K], p[K], v[K], d[K];
  int total = 0, ierr = 0;
  double res = 0.0;
  for (bool begun = false;; begun = true) {
    // r = b - A x in FP64; the barrier shows every block's x
    if (begun && !vg_sync(g, a.st)) return;
    double w[1];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = S.start + k * T + tid;
      double c[1] = {0.0};
      if (i < S.end) {
        const double ri = a.b[i] - row_spmv64<false>(a, a.x, i);
        a.r[i] = ri;
        c[0] = ri * ri;
      }
      resident_put<1>(S.cp, S.cps, k, c);
    }
    if (!resident_total<1>(S, g, a.st, w)) return;  // x is written again only after every block has read it
    const double rnorm = sqrt(w[0]);
    res = rnorm / bnrm;
    if (res <= a.tol) {
      write_result_m(a, g, total, res, 0);
      return;
    }
    if (begun && total >= a.maxit) {
      ierr = 1;
      break;
    }
    const double inv = 1.0 / rnorm;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = S.start + k * T + tid;
      r[k] = i < S.end ? (float)(a.r[i] * inv) : 0.0f;
      r0[k] = r[k];
      p[k] = v[k] = d[k] = 0.0f;
      const double c[1] = {(double)r[k] * (double)r[k]};
      resident_put<1>(S.cp, S.cps, k, c);
    }
    double w1[1];
    if (!resident_total<1>(S, g, a.st, w1)) return;
    const double target = m.tau * m.tau * w1[0];
    double rho_next = w1[0], rho_old = 1.0, alpha = 1.0, omega = 1.0;
    while (true) {
      ++total;
      const double rho = rho_next;
      if (fabs(rho) < DTINY) {
        ierr = 2;
        break;
      }
      const float beta = (float)((rho / rho_old) * (alpha / omega));
      const float om = (float)omega;
      float e[K];  // the exchanged vector: ph = D^-1 p, then sh = D^-1 s
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int l = k * T + tid;
        p[k] = fmaf(beta, fmaf(-om, v[k], p[k]), r[k]);
        e[k] = l < S.R ? resident_dinv<WC>(S, l) * p[k] : 0.0f;
      }
      if (!resident_exchange<WC, K>(S, e, a.st, [] {})) return;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int l = k * T + tid;
        float dinv;
        v[k] = l < S.R ? resident_row<WC>(S, l, dinv) : 0.0f;
        const double c[1] = {(double)r0[k] * (double)v[k]};
        resident_put<1>(S.cp, S.cps, k, c);
      }
      double d1[1];
      if (!resident_total<1>(S, g, a.st, d1)) return;
      alpha = rho / d1[0];
      const float af = (float)alpha;
      // r becomes s; d takes the half step (its other half follows after omega)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int l = k * T + tid;
        d[k] = fmaf(af, e[k], d[k]);
        r[k] = fmaf(-af, v[k], r[k]);
        e[k] = l < S.R ? resident_dinv<WC>(S, l) * r[k] : 0.0f;
        const double c[1] = {(double)r[k] * (double)r[k]};
        resident_put<1>(S.cp, S.cps, k, c);
      }
      if (!resident_exchange<WC, K>(S, e, a.st, [&] { total_post<1>(S, g); })) return;
      double d2[1];
      if (!total_wait<1>(S, g, a.st, d2)) return;
      if (d2[0] <= target || total >= a.maxit) break;
      float t[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int l = k * T + tid;
        float dinv;
        t[k] = l < S.R ? resident_row<WC>(S, l, dinv) : 0.0f;
        const double c[2] = {(double)t[k] * (double)t[k], (double)t[k] * (double)r[k]};
        resident_put<2>(S.cp, S.cps, k, c);
      }
      double d3[2];
      if (!resident_total<2>(S, g, a.st, d3)) return;
      if (d3[0] < DTINY) {
        ierr = 2;
        break;
      }
      omega = d3[1] / d3[0];
      if (fabs(omega) < DTINY) {
        ierr = 2;
        break;
      }
      const float omf = (float)omega;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        d[k] = fmaf(omf, e[k], d[k]);
        r[k] = fmaf(-omf, t[k], r[k]);
        const double c[2] = {(double)r[k] * (double)r[k], (double)r[k] * (double)r0[k]};
        resident_put<2>(S.cp, S.cps, k, c);
      }
      double d4[2];
      if (!resident_total<2>(S, g, a.st, d4)) return;
      if (d4[0] <= target || total >= a.maxit) break;
      rho_next = d4[1];
      rho_old = rho;
    }
    if (ierr == 2) break;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = S.start + k * T + tid;
      if (i < S.end) a.x[i] = fma(rnorm, (double)d[k], a.x[i]);
    }
  }
  write_result_m(a, g, total, res, ierr);
}

// Halo words of the block of R rows at R * blockIdx.x: the 32-row words outside
// its range that its columns touch; *most: the largest of all blocks. The
// window's flags in dynamic shared memory.
__global__ void k_halo_words(int n, int W, int ld, const int* __restrict__ ell_col, int bw, int R, int* most) {
  extern __shared__ unsigned flags[];
  const int s0 = blockIdx.x * R, e0 = s0 + R, wb = max(0, s0 - (bw + 31) / 32 * 32);
  const int nwords = (min(n, e0 + bw) - wb + 31) / 32;
  for (int w = threadIdx.x; w < nwords; w += blockDim.x) flags[w] = 0u;
  __syncthreads();
  for (int i = s0 + threadIdx.x; i < min(n, e0); i += blockDim.x)
    for (int t = 0; t < W; ++t) {
      const int c = ell_col[t * ld + i];
      if (c < s0 || c >= e0) flags[(c - wb) >> 5] = 1u;
    }
  __syncthreads();
  int mine = 0;
  for (int w = threadIdx.x; w < nwords; w += blockDim.x) mine += flags[w] != 0u;
  mine = __reduce_add_sync(0xffffffffu, mine);
  __shared__ int sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) atomicAdd(&sum, mine);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(most, sum);
}

enum { kBicg = 0, kPcg = 1, kPcgPaged = 2 };

// Threads of a block of R rows (a multiple of 256) and the rows of a thread,
// one of the compiled counts.
constexpr int block_threads(int R) { return R > kPairRows ? 512 : 256; }
constexpr int thread_rows(int R) {
  const int K = (R + block_threads(R) - 1) / block_threads(R);
  return K <= 5 ? K : K <= 7 ? 7 : 9;
}

constexpr int kPageMin = 5, kPageMax = 9;  // super-chunks of a page
constexpr int kPageThreadRows = thread_rows(kPageMin * kSuperRows);  // and the rows of its threads, at least
static_assert(block_threads(kPageMax * kSuperRows) == 256 && thread_rows(kPageMax * kSuperRows) == 9,
              "k_pcg_paged is compiled for blocks of 256 threads of up to 9 rows");

// The kernel of a solve; null when none is compiled for these rows a thread.
template <int WC, int K>
const void* resident_kernel_k(int which) {
  if (which == kBicg) return (const void*)k_bicgstab_resident<WC, K>;
  if (which == kPcg) return (const void*)k_pcg_resident<WC, K>;
  if constexpr (K >= kPageThreadRows) return (const void*)k_pcg_paged<WC, K>;
  return nullptr;
}

template <int WC>
const void* resident_kernel(int K, int which) {
  switch (K) {
    case 1: return resident_kernel_k<WC, 1>(which);
    case 2: return resident_kernel_k<WC, 2>(which);
    case 3: return resident_kernel_k<WC, 3>(which);
    case 4: return resident_kernel_k<WC, 4>(which);
    case 5: return resident_kernel_k<WC, 5>(which);
    case 7: return resident_kernel_k<WC, 7>(which);
    case 9: return resident_kernel_k<WC, 9>(which);
    default: return nullptr;
  }
}

constexpr int kStaticSmem = 4 * 1024;  // above the kernels' static shared memory and the driver's share of a block

int device_limits(int& sms, int& smem_sm) {
  int dev = 0;
  MGPU_CUDA(cudaGetDevice(&dev));
  MGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MGPU_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  return 0;
}

// The most halo words of a block when the rows are cut into blocks of R, and
// whether such a block fits: rows and window in an SM's shared memory, window
// offsets in 16 bits.
int fit_rows(int n, int W, int ld, const int* ell_col, int bw, int R, int room, int& words, bool& fits, int* most,
             cudaStream_t s) {
  const int WC = W <= 5 ? 5 : 7, flags = 4 * resident_window_words(R, bw);
  const int T = block_threads(R), K = thread_rows(R);
  fits = false;
  if (resident_smem(WC, R, bw, 0, K * (T / 32)) > room) return 0;
  if (flags + (int)sizeof(int) > 48 * 1024) return 0;  // with the kernel's own sum, a block's shared memory unasked
  MGPU_CUDA(cudaMemsetAsync(most, 0, sizeof(int), s));
  k_halo_words<<<(n + R - 1) / R, 256, flags, s>>>(n, W, ld, ell_col, bw, R, most);
  MGPU_CUDA(cudaGetLastError());
  MGPU_CUDA(cudaMemcpyAsync(&words, most, sizeof(int), cudaMemcpyDeviceToHost, s));
  MGPU_CUDA(cudaStreamSynchronize(s));
  fits = resident_smem(WC, R, bw, words, K * (T / 32)) <= room && 4 * (R + 32 * words) <= 65535;
  return 0;
}

// Bytes of a streamed polynomial step: ELL columns and values, the vectors of a pass.
double pass_bytes(int n, int W) { return (double)n * (8.0 * W + 56.0); }

// Below this many bytes a step the streamed solve still hits L2 and is the faster
// one whatever the pages' reach (hexahedra of 141 MB: 0.94 to 1.05 times as fast in
// turns, of 162 MB 1.06 to 1.17).
constexpr double kTurnBytes = 150e6;

// Whether a larger system is solved faster in turns than streamed; steps: page
// steps a block spends on a polynomial step of one page, loads and waits included.
// Both times of a polynomial step follow 65 systems timed both ways on several
// B200s. The streamed pass hardly differs between them; a page step, most of it
// exchange through L2, takes 3.6 to 5.0 us with 7 entries a row, 4.2 to 5.4 with 5. us
// an iteration, streamed / in turns, the fastest and the slowest seen: hexahedra in
// natural order, 1.44M rows 1,033 / 921, 975, 2.0M 1,541 / 1,234, 1,315, 4.1M 2,906 / 2,478,
// 2,643; in RCM order 2.0M 1,546 / 1,188, 1,276; mixed within 500 rows 1,650 / 1,790
// (refused); a 1000 x 2500 grid 1,569 / 974, 1,074; tetrahedra in natural order, 1.7M 1,030 /
// 1,049, 3.4M 2,034 / 2,289 (refused). Tetrahedra in RCM order lie on the line, 1.7M 1,022 /
// 983, 1,090, 3.07M 1,841 / 1,781, 2,060; a PISO step on the 3.07M took 220.8 / 211.1 ms,
// 216.9 / 213.8 on another GPU, its pressure solves 197.1 / 202.3 on a third.
bool turns_pay(int n, int W, int R, int blocks, double steps) {
  const bool wide = W > 5;
  const double streamed = pass_bytes(n, W) / (wide ? 7.3e6 : 7.6e6);  // us
  const double turns = std::ceil((double)n / R) / blocks + 0.5;  // the last turn has fewer pages than blocks
  return turns * steps * (wide ? 4.3 : 4.55) <= streamed;
}
}  // namespace

// Whether plan_resident may give pages to a system, by its size alone.
bool may_take_pages(int n, int W) { return W <= 7 && (g_resident_sms > 0 || pass_bytes(n, W) >= kTurnBytes); }

// The division of a system over the SMs for its resident solves: rows of a
// block (whole super-chunks) and the most halo words of a block; larger systems:
// the largest page and the steps of its turn. No plan (rows 0) with more than 7
// entries a row, or when the halo does not fit.
int plan_resident(int n, int W, int ld, const int* ell_col, int bw, ResidentPlan& plan, int* scratch, cudaStream_t s) {
  plan = ResidentPlan{};
  if (!ell_col || W > 7 || bw < 0 || n < kSuperRows / 4) return 0;
  int sms = 0, smem = 0;
  if (int e = device_limits(sms, smem)) return e;
  if (g_resident_sms > 0) sms = std::min(sms, g_resident_sms);
  const int nsc = (n + kSuperRows - 1) / kSuperRows;
  if (nsc > 256 * kSumGroups) return 0;
  const int pair = (nsc + 2 * sms - 1) / (2 * sms), single = (nsc + sms - 1) / sms;
  const int half = smem / 2 - kStaticSmem, whole = smem - kStaticSmem;
  int words = 0;
  bool fits = false;
  auto keep = [&](int R) {
    plan.rows = R;
    plan.words = words;
    plan.bw = bw;
    plan.blocks = std::min((n + R - 1) / R, 2 * sms);
  };
  // two blocks of 256 threads per SM up to 6 super-chunks each (one PCG
  // iteration of 42,253 rows 42 -> 35 us against one block of 512), then one of
  // 512 (524,288 rows: 116 us against 121 for two of 256)
  if (pair <= 6) {
    if (int e = fit_rows(n, W, ld, ell_col, bw, pair * kSuperRows, half, words, fits, scratch, s)) return e;
    if (fits) keep(pair * kSuperRows);
    if (fits) return 0;
  }
  if (single * kSuperRows > kPairRows && single <= 18) {
    if (int e = fit_rows(n, W, ld, ell_col, bw, single * kSuperRows, whole, words, fits, scratch, s)) return e;
    if (fits) keep(single * kSuperRows);
    if (fits) return 0;
  }
  if (!may_take_pages(n, W)) return 0;
  // pages: the largest that fits in half an SM, and the steps that make the most
  // of the shared memory. With G blocks, r pages of reach and a load that takes as
  // long as L = 2 steps, steps pass at s (G - (s - 1) r) / (L + s) pages a step time
  // (each page waits (s - 1) r pages' worth for those ahead of it).
  const int most = 2 * sms;
  for (int sc = kPageMax; sc >= kPageMin && !fits; --sc) {
    const int R = sc * kSuperRows;
    if (R * (long)most > n) continue;  // a page for every block at least
    if (int e = fit_rows(n, W, ld, ell_col, bw, R, half, words, fits, scratch, s)) return e;
    if (!fits) continue;
    const double r = (double)bw / R;
    double best = 0.0;
    for (int st = 2; st <= 16 && 2 * (st - 1) * (int)std::ceil(r) < most; ++st) {
      const double rate = st * (most - (st - 1) * r) / (2.0 + st);
      if (rate > best) {
        best = rate;
        plan.steps = st;
      }
    }
    if (best <= 0.0 || (g_resident_sms == 0 && !turns_pay(n, W, R, most, most / best))) {
      plan = ResidentPlan{};
      return 0;
    }
    keep(R);
  }
  return 0;
}

// Floats that a plan's pages take after the FP32 CSR values (MixedArgs::a32).
size_t page_floats(int n, int W, const ResidentPlan& plan) {
  if (plan.steps == 0) return 0;
  return (size_t)page_bytes(W <= 5 ? 5 : 7, plan.rows, plan.words) / 4 * ((n + plan.rows - 1) / plan.rows) + 32;
}

// The resident solve of a planned system; *taken = false and no launch when
// there is no plan, no polynomial to apply, no kernel for the plan's rows, or
// turns are planned (pressure only). A planned system always takes it. Measured
// against the streaming kernel from 64 rows (the smallest planned) to the largest
// that fits, about 570,000 rows of 7 entries and 680,000 of 5: 1.6 to 3 times as
// fast in natural and RCM order, mixed within 500, 1,500, 3,000 and 6,000 rows 1.3-2.0,
// 1.1-1.8, 1.1-1.6 and 1.0-1.3 where the halo fits (a BiCGStab iteration 1.2-1.8).
int launch_resident(const KrylovArgs& a, const MixedArgs& m, bool pcg, cudaStream_t s, bool* taken) {
  *taken = false;
  if (m.plan.rows <= 0 || (pcg && (!m.ell64 || m.cheb_k < 2 || m.cheb_k > 64))) return 0;
  const bool paged = m.plan.steps > 0;
  if (paged && !pcg) return 0;
  const int R = m.plan.rows, WC = m.ell_w <= 5 ? 5 : 7;
  const int T = block_threads(R), K = thread_rows(R);
  const int dyn = resident_smem(WC, R, m.plan.bw, m.plan.words, K * (T / 32));
  const int which = paged ? kPcgPaged : pcg ? kPcg : kBicg;
  const void* fn = WC == 5 ? resident_kernel<5>(K, which) : resident_kernel<7>(K, which);
  if (!fn) return 0;
  int sms = 0, smem = 0;
  if (int e = device_limits(sms, smem)) return e;
  // the same limit on every call: another thread may be launching the kernel for another system
  MGPU_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem - kStaticSmem));
  KrylovArgs aa = a;
  MixedArgs mm = m;
  int RR = R, words = m.plan.words;
  WaitLimits waits = wait_limits(g_spin_limit, g_exchange_limit);
  void* args[] = {&aa, &mm, &waits, &RR, &words};  // the paged kernel takes the first three
  MGPU_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned long long), s));
  MGPU_CUDA(cudaLaunchCooperativeKernel(fn, dim3(m.plan.blocks), dim3(T), args, (size_t)dyn, s));
  *taken = true;
  return 0;
}

}  // namespace mgpu
