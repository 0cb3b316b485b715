// krylov_sweep.cu -- the FP64 parity form's ILU(0) / IC(0) solves on rows that
// stay in shared memory: cg_ic0 and PCG+ILU(0), bicgstab_ilu0
// (mod_uns_linsolver.f90:148-224, 405-461), the same bits as krylov.cu's.
//
// What bounds these solves is the serial chain of the triangular sweeps: one hop
// per level, some 250 levels an iteration on a few thousand rows. In krylov.cu a
// hop is a chain of trips to L1 or L2: the row number, its pointers, its factor
// values, the neighbours' results, a block barrier or a poll of a value another
// block stores (0.9 us in one block, 2.6 us between blocks). Here a block owns a
// contiguous range of rows (as few blocks as shared memory allows: a hop inside
// a block is several times shorter than one between blocks) and keeps their
// factor rows, level lists and the swept vector in shared memory. A hop inside
// it is straight-line code: the neighbours' values from shared memory, the row's
// operations, a barrier of the warps that the widest level needs, with the next
// level's row already in registers. The values of other blocks (rows within a
// bandwidth of the range) are brought into shared memory by warps of their own,
// which poll the exchange words (exchange.cuh) that those blocks write. Rows are
// taken in level order on every block, so the least unfinished row can always
// proceed: the blocks are co-resident and a sweep ends.
//
// The dot products keep krylov.cu's order for the grid it would have launched:
// the rows' products go to global memory and are added by the threads that
// stand for that grid's (grid_sum).
//
// Measured on a B200, one PCG iteration (krylov.cu -> here): IC(0) on the 64 x 64
// cavity (254 levels, 2 blocks) 240 -> 92 us, on 32^3 cells (15 blocks) 600 ->
// 130 us, ILU(0) on a 65,536-cell channel (RCM order, 29 blocks) 660 -> 290 us. A
// level costs about 0.3 us with one warp (the FP64 chain of the row: a product and
// a subtraction an entry, four operations of the quotient), 0.9 us with a thousand
// rows. 1024 threads (64 registers) were 17 % slower on the cavity and equal on the
// channel.

#include <algorithm>

#include "exchange.cuh"

namespace mgpu {
extern unsigned g_spin_limit;      // krylov.cu: the spin_limit tuning key
extern unsigned g_exchange_limit;  // krylov.cu: the exchange_spin_limit tuning key
namespace {

constexpr int kSweepThreads = 512;
constexpr int kPollWarps = 4;  // at least; the warps that no level needs poll too

// Marks a value that has not arrived: a signalling NaN, which arithmetic never yields.
constexpr unsigned long long kPending = 0x7FF0DEAD0BADF00Dull;

// A block's rows: sizes, and byte offsets into its shared memory. W: most
// entries of a row on one side of the diagonal. A side's arrays are in its level
// order, each row's entries in the order they apply and padded with (0, the
// zero), so that a row is read and applied without a branch.
template <int W>
struct Sweep {
  static constexpr int CW = W <= 4 ? 4 : 8;  // places a row
  int n, R, start, end;
  int bw;            // largest |column - row|
  int kind;          // 0 ILU(0), 2 IC(0)
  double* prod;      // per-row products of the sums (2 halves x 2 sums), see products()
  double* part;      // krylov.cu's per-block partial sums (2 halves x 2 sums x vgrid)
  int vgrid;         // krylov.cu's grid: one block of 512 threads, or vgrid of 256
  unsigned sums;     // sums so far
  unsigned aseq;     // applications so far
  u64 *fwd, *bwd;    // exchange words (pairs) of the forward and backward results
  int w;             // double: the swept vector [0, R), a zero at R, the other blocks' values at [-bw, 0)
  int fd, fy;        // double[R]: factor diagonal and its reciprocal, by row
  struct Side {
    int f;           // double[W][R]: factor entries (IC(0)'s upper side: of the transposed factor)
    int c;           // unsigned short[R][CW]: where their values are, from the first of the other blocks' values
    int l;           // unsigned short[R]: row; kPublish: another block may need its value
    int p;           // unsigned short[R + 1]: first of each local level
    int nlev;        // local levels (those with a row of this block)
  } lo, up;
  int warps;         // warps that the widest of them needs
  WaitLimits waits;
};
constexpr unsigned kPublish = 0x8000u;

constexpr int sweep_row_bytes(int W) { return 24 + 2 * (8 * W + 2 * (W <= 4 ? 4 : 8) + 4); }
inline long sweep_smem(int W, int R, int bw) { return (long)sweep_row_bytes(W) * R + 8l * bw + 64; }

template <int W>
__device__ __forceinline__ void sweep_views(Sweep<W>& S, int R, int bw) {
  S.R = R;
  S.w = 8 * bw;
  S.fd = S.w + 8 * (R + 1);
  S.fy = S.fd + 8 * R;
  int at = (S.fy + 8 * R + 15) & ~15;
  auto side = [&](typename Sweep<W>::Side& d) {
    d.c = at;
    d.f = d.c + 2 * Sweep<W>::CW * R;
    at = d.f + 8 * W * R;
  };
  side(S.lo);
  side(S.up);
  S.lo.l = at;
  S.up.l = S.lo.l + 2 * R;
  S.lo.p = S.up.l + 2 * R;
  S.up.p = S.lo.p + 2 * (R + 1);
}

// the products of the next sum (n; those of a second one n further on): z and w,
// or the space after the exchange words
template <int W>
__device__ __forceinline__ double* products(const Sweep<W>& S) {
  return S.prod + (S.sums & 1u) * 6l * S.n;
}

// The block's rows of a level order (ptr, rows: the system's, rows ascending in
// a level) as local lists; returns the number of local levels. scratch: int[2 * R]
// in shared memory.
__device__ __forceinline__ int local_levels(const int* __restrict__ ptr, const int* __restrict__ rows, int nlev,
                                            int start, int end, int out, int lptr, int scratch, int& widest) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  __shared__ int s_cnt[32], s_lev[32], s_base[2];
  if (tid == 0) s_base[0] = s_base[1] = 0;
  __syncthreads();
  for (int l0 = 0; l0 < nlev; l0 += blockDim.x) {
    const int lev = l0 + tid;
    int lb = 0, cnt = 0;
    if (lev < nlev) {
      const int b = ptr[lev], e = ptr[lev + 1];
      auto below = [&](int key) {
        int lo = b, hi = e;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (rows[mid] < key)
            lo = mid + 1;
          else
            hi = mid;
        }
        return lo;
      };
      lb = below(start);
      cnt = below(end) - lb;
    }
    // exclusive prefix of (rows, non-empty levels) over the block
    int c = cnt, v = cnt > 0 ? 1 : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, c, o), d = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) {
        c += a;
        v += d;
      }
    }
    if (lane == 31) {
      s_cnt[warp] = c;
      s_lev[warp] = v;
    }
    __syncthreads();
    int rbase = s_base[0], lbase = s_base[1];
    for (int q = 0; q < warp; ++q) {
      rbase += s_cnt[q];
      lbase += s_lev[q];
    }
    if (cnt > 0) {
      const int k = lbase + v - 1;
      smem_at<unsigned short>(lptr, k) = (unsigned short)(rbase + c - cnt);
      smem_at<int>(scratch, 2 * k) = lb;
      smem_at<int>(scratch, 2 * k + 1) = cnt;
    }
    __syncthreads();
    if (tid == (int)blockDim.x - 1) {
      s_base[0] = rbase + c;
      s_base[1] = lbase + v;
    }
    __syncthreads();
  }
  const int nl = s_base[1];
  if (tid == 0) smem_at<unsigned short>(lptr, nl) = (unsigned short)s_base[0];
  for (int k = warp; k < nl; k += nw) {
    const int lb = smem_at<int>(scratch, 2 * k), cnt = smem_at<int>(scratch, 2 * k + 1);
    const int to = smem_at<unsigned short>(lptr, k);
    for (int j = lane; j < cnt; j += 32) smem_at<unsigned short>(out, to + j) = (unsigned short)(rows[lb + j] - start);
  }
  int most = 0;
  for (int k = lane; k < nl; k += 32) most = max(most, smem_at<int>(scratch, 2 * k + 1));
  widest = max(widest, __reduce_max_sync(0xffffffffu, most));
  __syncthreads();
  return nl;
}

// A side's rows in its level order: entries, places, and the rows that other
// blocks may need (those within a bandwidth of the range's end or start).
template <int W, bool LOWER>
__device__ __forceinline__ void side_rows(const KrylovArgs& a, const Sweep<W>& S) {
  const typename Sweep<W>::Side& d = LOWER ? S.lo : S.up;
  const int rows = S.end - S.start;
  for (int idx = threadIdx.x; idx < rows; idx += blockDim.x) {
    const int l = smem_at<unsigned short>(d.l, idx), i = S.start + l;
    const int di = a.diag[i], k0 = LOWER ? a.row_ptr[i] : di + 1, k1 = LOWER ? di : a.row_ptr[i + 1];
#pragma unroll
    for (int t = 0; t < W; ++t) {
      const bool in = k0 + t < k1;
      // IC(0)'s backward sweep applies the entries in descending column order
      const int k = !LOWER && S.kind == 2 ? k1 - 1 - t : k0 + t;
      int place = S.bw + S.R;
      double f = 0.0;
      if (in) {
        f = a.fval[!LOWER && S.kind == 2 ? a.lt_pos[k] : k];
        const int c = a.col[k] - S.start;
        // the rows after the range share the places of those before it
        place = (unsigned)c < (unsigned)S.R ? S.bw + c : LOWER ? S.bw + c : c - S.R;
      }
      smem_at<double>(d.f, t * S.R + idx) = f;
      smem_at<unsigned short>(d.c, idx * Sweep<W>::CW + t) = (unsigned short)place;
    }
    const bool out = LOWER ? l + S.bw >= rows && S.end < S.n : l < S.bw && S.start > 0;
    if (out) smem_at<unsigned short>(d.l, idx) = (unsigned short)(l | kPublish);
  }
}

// The block's part of the system in shared memory, its words cleared; the
// barrier puts every block's clears (and zeroed x) before what follows.
template <int W>
__device__ __forceinline__ bool sweep_prologue(const KrylovArgs& a, VGrid& g, Sweep<W>& S) {
  int widest = 0;
  S.lo.nlev = local_levels(a.lo_ptr, a.lo_rows, a.nlev_lo, S.start, S.end, S.lo.l, S.lo.p, S.lo.f, widest);
  S.up.nlev = local_levels(a.up_ptr, a.up_rows, a.nlev_up, S.start, S.end, S.up.l, S.up.p, S.lo.f, widest);
  S.warps = min((widest + 31) / 32, (int)(blockDim.x >> 5) - kPollWarps);
  for (int i = S.start + threadIdx.x; i < S.end; i += blockDim.x) {
    const double d = a.fval[a.diag[i]];
    smem_at<double>(S.fd, i - S.start) = d;
    smem_at<double>(S.fy, i - S.start) = 1.0 / d;
    S.fwd[2l * i] = S.fwd[2l * i + 1] = 0ull;
    S.bwd[2l * i] = S.bwd[2l * i + 1] = 0ull;
    if (a.zero_x) a.x[i] = 0.0;
  }
  side_rows<W, true>(a, S);
  side_rows<W, false>(a, S);
  if (threadIdx.x == 0) smem_at<double>(S.w, S.R) = 0.0;
  return vg_sync(g, a.st);
}

// s / d from y = 1 / d rounded to nearest: two corrections of the quotient by
// its exact remainder (P. Markstein, Computation of elementary functions on the
// IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990: with y correctly
// rounded and q within an ulp, q + (s - q d) y rounds to the quotient). Only
// these four operations wait for s. Outside the exponents where no intermediate
// can over- or underflow, the division itself.
__device__ __forceinline__ double quotient(double s, double d, double y) {
  const int es = (__double2hiint(s) >> 20) & 0x7ff, ed = (__double2hiint(d) >> 20) & 0x7ff;
  double q = s * y;
  q = fma(fma(-d, q, s), y, q);
  q = fma(fma(-d, q, s), y, q);
  const bool plain = (unsigned)(es - 512) < 1024u && (unsigned)(ed - 800) < 448u;
  return plain ? q : s / d;
}

// A row of the next level, read ahead of the barrier before it.
template <int W>
struct Fetched {
  unsigned l;    // its number, with kPublish
  double f[W];
  unsigned c[W];  // byte offsets of the values
};

template <int W>
__device__ __forceinline__ void fetch_row(const Sweep<W>& S, const typename Sweep<W>::Side& d, int idx,
                                          Fetched<W>& r) {
  r.l = smem_at<unsigned short>(d.l, idx);
  unsigned pk[Sweep<W>::CW / 2];
  if constexpr (W <= 4) {
    const uint2 c = smem_at<uint2>(d.c, idx);
    pk[0] = c.x;
    pk[1] = c.y;
  } else {
    const uint4 c = smem_at<uint4>(d.c, idx);
    pk[0] = c.x;
    pk[1] = c.y;
    pk[2] = c.z;
    pk[3] = c.w;
  }
#pragma unroll
  for (int t = 0; t < W; ++t) {
    r.f[t] = smem_at<double>(d.f, t * S.R + idx);
    r.c[t] = t & 1 ? pk[t / 2] >> 16 : pk[t / 2] & 0xffffu;
  }
}

__device__ __forceinline__ double ld_value(unsigned place) {
  double v;
  const unsigned at = (unsigned)__cvta_generic_to_shared(block_smem) + 8u * place;
  asm volatile("ld.relaxed.cta.shared.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void st_value(unsigned place, double v) {
  const unsigned at = (unsigned)__cvta_generic_to_shared(block_smem) + 8u * place;
  asm volatile("st.relaxed.cta.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
__device__ __forceinline__ bool pending(double v) { return (u64)__double_as_longlong(v) == kPending; }

template <int W, bool FWD>
__device__ __forceinline__ bool sweep_row(const Sweep<W>& S, const Fetched<W>& r, DevStatus* st) {
  const unsigned l = r.l & (kPublish - 1u);
  double v[W], d = 1.0, y = 1.0;
  bool ok = true, wait = false;
#pragma unroll
  for (int t = 0; t < W; ++t) v[t] = ld_value(r.c[t]);
  double s = ld_value(S.bw + l);
  const bool divide = !FWD || S.kind == 2;
  if (divide) {
    d = smem_at<double>(S.fd, l);
    y = smem_at<double>(S.fy, l);
  }
#pragma unroll
  for (int t = 0; t < W; ++t) wait = wait || pending(v[t]);
  if (wait) {
    unsigned polls = S.waits.shared;
#pragma unroll
    for (int t = 0; t < W; ++t)
      while (pending(v[t]) && ok) {
        ok = keep_polling(polls, st);
        v[t] = ld_value(r.c[t]);
      }
  }
#pragma unroll
  for (int t = 0; t < W; ++t) s = s - r.f[t] * v[t];
  if (divide) s = quotient(s, d, y);
  st_value(S.bw + l, s);
  if (r.l & kPublish) st_pair((FWD ? S.fwd : S.bwd) + 2l * (S.start + (int)l), s, S.aseq);
  return ok;
}

// The levels in order, by the first S.warps warps; bar.sync 1 is theirs.
template <int W, bool FWD>
__device__ __forceinline__ bool sweep_levels(const Sweep<W>& S, DevStatus* st) {
  const typename Sweep<W>::Side& d = FWD ? S.lo : S.up;
  const int tid = threadIdx.x, T = 32 * S.warps, nlev = d.nlev, rows = S.end - S.start;
  bool ok = true;
  Fetched<W> r;
  int b = tid, e = smem_at<unsigned short>(d.p, 1), e1 = smem_at<unsigned short>(d.p, min(2, nlev));
  fetch_row<W>(S, d, min(b, rows - 1), r);
  for (int lev = 0; lev < nlev; ++lev) {
    if (b < e) ok = sweep_row<W, FWD>(S, r, st) && ok;
    for (int idx = b + T; idx < e; idx += T) {
      fetch_row<W>(S, d, idx, r);
      ok = sweep_row<W, FWD>(S, r, st) && ok;
    }
    b = e + tid;
    e = e1;
    e1 = smem_at<unsigned short>(d.p, min(lev + 3, nlev));
    fetch_row<W>(S, d, min(b, rows - 1), r);
    asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory");
  }
  return ok;
}

// The other warps: the values of the rows before the range (forward) or after it
// (backward) as their blocks write them, each thread taking its rows in turn
// without waiting for any one of them.
template <int W, bool FWD>
__device__ __forceinline__ bool sweep_poll(const Sweep<W>& S, DevStatus* st) {
  const int P = (int)blockDim.x - 32 * S.warps, tid = (int)threadIdx.x - 32 * S.warps;
  const u64* words = FWD ? S.fwd : S.bwd;
  const int first = FWD ? S.start - S.bw : S.end;  // row of place -bw
  unsigned left = 0u;
  for (int k = 0, j = tid; j < S.bw; j += P, ++k)
    if (first + j >= 0 && first + j < S.n) left |= 1u << k;
  unsigned polls = S.waits.value;
  while (left) {
    for (unsigned m = left; m; m &= m - 1u) {
      const int k = __ffs(m) - 1, j = tid + k * P;
      u64 lo, hi;
      ld_pair(words + 2l * (first + j), lo, hi);
      if ((unsigned)(lo >> 32) == S.aseq && (unsigned)(hi >> 32) == S.aseq) {
        st_value(j, __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull))));
        left &= ~(1u << k);
      }
    }
    if (left && !keep_polling(polls, st)) return false;
  }
  return true;
}

template <int W, bool FWD>
__device__ __forceinline__ bool sweep_half(const Sweep<W>& S, DevStatus* st) {
  for (int j = threadIdx.x; j < S.bw; j += blockDim.x)
    st_value(j, __longlong_as_double((long long)kPending));
  __syncthreads();
  const bool ok = (int)threadIdx.x < 32 * S.warps ? sweep_levels<W, FWD>(S, st) : sweep_poll<W, FWD>(S, st);
  return __syncthreads_and(ok) != 0;
}

// dst = M^-1 src on the block's rows. The words of an application are written
// again only after a sum or barrier over all blocks, which each block joins when
// it has read all it needs.
template <int W>
__device__ __forceinline__ bool sweep_apply(Sweep<W>& S, const double* src, double* dst, DevStatus* st) {
  const int n = S.end - S.start;
  ++S.aseq;
  for (int l = threadIdx.x; l < n; l += blockDim.x) smem_at<double>(S.w, l) = src[S.start + l];
  if (!sweep_half<W, true>(S, st) || !sweep_half<W, false>(S, st)) return false;
  for (int l = threadIdx.x; l < n; l += blockDim.x) dst[S.start + l] = smem_at<double>(S.w, l);
  return true;
}

// y_i = A_i . x in csr_matvec order, the row's first 8 loads issued together
__device__ __forceinline__ double row_product(const KrylovArgs& a, const double* x, int i) {
  const int b = a.row_ptr[i], e = a.row_ptr[i + 1];
  double v[8], xv[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    v[t] = xv[t] = 0.0;
    if (b + t < e) {
      v[t] = a.aval[b + t];
      xv[t] = ldv(&x[a.col[b + t]]);
    }
  }
  double y = 0.0;
#pragma unroll
  for (int t = 0; t < 8; ++t)
    if (b + t < e) y = y + v[t] * xv[t];
  for (int k = b + 8; k < e; ++k) y = y + a.aval[k] * ldv(&x[a.col[k]]);
  return y;
}

__device__ __forceinline__ void sweep_result(const KrylovArgs& a, int it, double res, int ierr) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  MgpuIterRec* rec = a.recs + a.st->cur_it;
  if (a.slot >= 0 && a.slot < MGPU_MAXSOLVE) {
    rec->lin_it[a.slot] = it;
    rec->lin_res[a.slot] = res;
    rec->lin_ierr[a.slot] = ierr;
    if (rec->nsolve < a.slot + 1) rec->nsolve = a.slot + 1;
  }
  if (ierr == 2 && a.ier_breakdown != 0) {
    a.st->ier = a.ier_breakdown;
    a.st->abort = 1;
  }
}

// The sums of the products (every block has written its
// rows') in the order of krylov.cu's vg_sum: on one block of 512 threads each
// adds its rows in steps of 512, then butterflies over the warps and over the 16
// warp sums; on vgrid blocks of 256, each thread its rows in steps of the grid,
// butterflies within its block, and the blocks' partial sums in a fixed order of
// 256 threads. Every block of this launch computes all (the partials: its share).
template <int NQ, int W>
__device__ __forceinline__ bool grid_sum(Sweep<W>& S, VGrid& g, DevStatus* st, double (&out)[NQ]) {
  __shared__ double s_warp[2][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned half = S.sums & 1u;
  const double* c = products(S);
  ++S.sums;
  if (!vg_sync(g, st)) return false;
  if (S.vgrid == 1) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double v = 0.0;
#pragma unroll 8
      for (int i = tid; i < S.n; i += 512) v = v + ldv(&c[(long)q * S.n + i]);
      v = warp_sum(v);
      if (lane == 0) s_warp[q][warp] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) out[q] = warp_sum(lane < 16 ? s_warp[q][lane] : 0.0);
    __syncthreads();
    return true;
  }
  const int vb = S.vgrid, step = 256 * vb;
  double* part = S.part + half * 2l * vb;
  for (int b0 = 2 * g.rank; b0 < vb; b0 += 2 * g.nb) {
    const int b = b0 + (tid >> 8);  // two of its blocks side by side
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double v = 0.0;
      if (b < vb)
        for (int i = 256 * b + (tid & 255); i < S.n; i += step) v = v + ldv(&c[(long)q * S.n + i]);
      v = warp_sum(v);
      if (lane == 0) s_warp[q][warp] = v;
    }
    __syncthreads();
    if ((warp & 7) == 0 && b < vb) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double v = warp_sum(lane < 8 ? s_warp[q][warp + lane] : 0.0);
        if (lane == 0) part[(long)q * vb + b] = v;
      }
    }
    __syncthreads();
  }
  if (!vg_sync(g, st)) return false;
  if (warp < 8) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const double* p = part + (long)q * vb;
      double t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;
      if (tid < vb) t0 = ldv(&p[tid]);
      if (tid + 256 < vb) t1 = ldv(&p[tid + 256]);
      if (tid + 512 < vb) t2 = ldv(&p[tid + 512]);
      if (tid + 768 < vb) t3 = ldv(&p[tid + 768]);
      double v = ((t0 + t1) + t2) + t3;
      for (int j = tid + 1024; j < vb; j += 256) v = v + ldv(&p[j]);
      v = warp_sum(v);
      if (lane == 0) s_warp[q][warp] = v;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) out[q] = warp_sum(lane < 8 ? s_warp[q][lane] : 0.0);
  __syncthreads();
  return true;
}

template <int W>
__device__ __forceinline__ void sweep_begin(const KrylovArgs& a, const VGrid& g, Sweep<W>& S, int R, int vgrid,
                                            WaitLimits waits) {
  S.waits = waits;
  S.n = a.n;
  S.bw = a.bw;
  S.kind = a.precond;
  S.start = g.rank * R;
  S.end = min(a.n, S.start + R);
  S.aseq = S.sums = 0u;
  double* more = a.w + a.n;  // 6 n more than krylov.cu's work vectors
  S.fwd = reinterpret_cast<u64*>(more);
  S.bwd = reinterpret_cast<u64*>(more + 2l * a.n);
  S.prod = a.z;
  S.part = a.partials;
  S.vgrid = vgrid;
  sweep_views<W>(S, R, a.bw);
}

#define MGPU_OWN_ROWS(i) for (int i = S.start + (int)threadIdx.x; i < S.end; i += (int)blockDim.x)

// k_pcg (krylov.cu) with ILU(0) or IC(0). LIMITS: the waits' limits are those of the
// launch (the tuning keys); compiled in otherwise, as with limits at run time the
// compiler's code took 317 us instead of 283 an iteration on the 64 x 32 x 32 box.
template <int W, bool LIMITS>
__global__ void __launch_bounds__(kSweepThreads, 1) k_pcg_sweep(KrylovArgs a, int R, int vgrid, WaitLimits waits) {
  if (a.st->abort) return;
  VGrid g = whole_grid(a.bar, a.partials, true);
  Sweep<W> S;
  sweep_begin<W>(a, g, S, R, vgrid, LIMITS ? waits : wait_limits(0u, 0u));
  double *x = a.x, *r = a.r, *p = a.p, *q = a.v, *z = a.r0;
  if (!sweep_prologue<W>(a, g, S)) return;
  double t[1];
  MGPU_OWN_ROWS(i) products(S)[i] = a.b[i] * a.b[i];
  if (!grid_sum<1>(S, g, a.st, t)) return;
  const double bnrm = sqrt(t[0]);
  if (bnrm == 0.0) {
    MGPU_OWN_ROWS(i) x[i] = 0.0;
    sweep_result(a, 0, 0.0, 0);
    return;
  }
  if (*a.ferr != 0) {
    sweep_result(a, 0, 0.0, *a.ferr + 10);
    return;
  }
  MGPU_OWN_ROWS(i) {
    const double ri = a.b[i] - row_product(a, x, i);
    r[i] = ri;
    products(S)[i] = ri * ri;
  }
  if (!grid_sum<1>(S, g, a.st, t)) return;
  double res = sqrt(t[0]) / bnrm;
  if (res <= a.tol) {
    sweep_result(a, 0, res, 0);
    return;
  }
  if (!sweep_apply(S, r, z, a.st)) return;
  MGPU_OWN_ROWS(i) {
    const double zi = z[i];
    p[i] = zi;
    products(S)[i] = r[i] * zi;
  }
  if (!grid_sum<1>(S, g, a.st, t)) return;  // its barrier shows every block's p
  double rz = t[0];
  int ierr = 0, it;
  for (it = 1; it <= a.maxit; ++it) {
    MGPU_OWN_ROWS(i) {
      const double qi = row_product(a, p, i);
      q[i] = qi;
      products(S)[i] = p[i] * qi;
    }
    if (!grid_sum<1>(S, g, a.st, t)) return;
    const double pap = t[0];
    if (fabs(pap) < DTINY) {
      ierr = 2;
      break;
    }
    const double alpha = rz / pap;
    MGPU_OWN_ROWS(i) {
      x[i] = x[i] + alpha * p[i];
      const double ri = r[i] - alpha * q[i];
      r[i] = ri;
      products(S)[i] = ri * ri;
    }
    if (!grid_sum<1>(S, g, a.st, t)) return;
    res = sqrt(t[0]) / bnrm;
    if (res <= a.tol) {
      sweep_result(a, it, res, 0);
      return;
    }
    if (!sweep_apply(S, r, z, a.st)) return;
    MGPU_OWN_ROWS(i) products(S)[i] = r[i] * z[i];
    if (!grid_sum<1>(S, g, a.st, t)) return;
    if (fabs(rz) < DTINY) {
      ierr = 2;
      break;
    }
    const double beta = t[0] / rz;
    MGPU_OWN_ROWS(i) p[i] = z[i] + beta * p[i];
    if (!vg_sync(g, a.st)) return;
    rz = t[0];
  }
  if (ierr == 0) ierr = 1;
  sweep_result(a, it, res, ierr);
}

// k_bicgstab (krylov.cu) with ILU(0)
template <int W, bool LIMITS>
__global__ void __launch_bounds__(kSweepThreads, 1) k_bicgstab_sweep(KrylovArgs a, int R, int vgrid, WaitLimits waits) {
  if (a.st->abort) return;
  VGrid g = whole_grid(a.bar, a.partials, true);
  Sweep<W> S;
  sweep_begin<W>(a, g, S, R, vgrid, LIMITS ? waits : wait_limits(0u, 0u));
  double *x = a.x, *r = a.r, *r0 = a.r0, *p = a.p, *v = a.v, *s = a.s, *t = a.t, *ph = a.ph, *sh = a.sh;
  if (!sweep_prologue<W>(a, g, S)) return;
  double t1[1];
  MGPU_OWN_ROWS(i) products(S)[i] = a.b[i] * a.b[i];
  if (!grid_sum<1>(S, g, a.st, t1)) return;
  const double bnrm = sqrt(t1[0]);
  if (bnrm == 0.0) {
    MGPU_OWN_ROWS(i) x[i] = 0.0;
    sweep_result(a, 0, 0.0, 0);
    return;
  }
  if (*a.ferr != 0) {
    sweep_result(a, 0, 0.0, *a.ferr + 10);
    return;
  }
  MGPU_OWN_ROWS(i) {
    const double ri = a.b[i] - row_product(a, x, i);
    r0[i] = ri;
    r[i] = ri;
    p[i] = 0.0;
    v[i] = 0.0;
    products(S)[i] = ri * ri;
  }
  if (!grid_sum<1>(S, g, a.st, t1)) return;
  double res = sqrt(t1[0]) / bnrm;
  if (res <= a.tol) {
    sweep_result(a, 0, res, 0);
    return;
  }
  double rho_next = t1[0], rho_old = 1.0, alpha = 1.0, omega = 1.0;
  int ierr = 0, it;
  for (it = 1; it <= a.maxit; ++it) {
    const double rho = rho_next;
    if (fabs(rho) < DTINY) {
      ierr = 2;
      break;
    }
    const double beta = (rho / rho_old) * (alpha / omega);
    MGPU_OWN_ROWS(i) p[i] = r[i] + beta * (p[i] - omega * v[i]);
    if (!sweep_apply(S, p, ph, a.st)) return;
    if (!vg_sync(g, a.st)) return;
    MGPU_OWN_ROWS(i) {
      const double vi = row_product(a, ph, i);
      v[i] = vi;
      products(S)[i] = r0[i] * vi;
    }
    if (!grid_sum<1>(S, g, a.st, t1)) return;
    alpha = rho / t1[0];
    MGPU_OWN_ROWS(i) {
      const double si = r[i] - alpha * v[i];
      s[i] = si;
      products(S)[i] = si * si;
    }
    if (!grid_sum<1>(S, g, a.st, t1)) return;
    const double snrm = sqrt(t1[0]);
    if (snrm / bnrm <= a.tol) {
      MGPU_OWN_ROWS(i) x[i] = x[i] + alpha * ph[i];
      sweep_result(a, it, snrm / bnrm, 0);
      return;
    }
    if (!sweep_apply(S, s, sh, a.st)) return;
    if (!vg_sync(g, a.st)) return;
    MGPU_OWN_ROWS(i) {
      const double ti = row_product(a, sh, i);
      t[i] = ti;
      products(S)[i] = ti * ti;
      products(S)[S.n + i] = ti * s[i];
    }
    double t2[2];
    if (!grid_sum<2>(S, g, a.st, t2)) return;
    const double tt = t2[0];
    if (tt < DTINY) {
      ierr = 2;
      break;
    }
    omega = t2[1] / tt;
    if (fabs(omega) < DTINY) {
      ierr = 2;
      break;
    }
    MGPU_OWN_ROWS(i) {
      x[i] = x[i] + alpha * ph[i] + omega * sh[i];
      const double ri = s[i] - omega * t[i];
      r[i] = ri;
      products(S)[i] = ri * ri;
      products(S)[S.n + i] = ri * r0[i];
    }
    if (!grid_sum<2>(S, g, a.st, t2)) return;
    res = sqrt(t2[0]) / bnrm;
    if (res <= a.tol) {
      sweep_result(a, it, res, 0);
      return;
    }
    rho_next = t2[1];
    rho_old = rho;
  }
  if (ierr == 0) {
    ierr = 1;
    it = a.maxit;
  }
  sweep_result(a, it, res, ierr);
}
#undef MGPU_OWN_ROWS

}  // namespace

template <int W>
const void* sweep_kernel(bool pcg, bool limits) {
  if (limits) return pcg ? (const void*)k_pcg_sweep<W, true> : (const void*)k_bicgstab_sweep<W, true>;
  return pcg ? (const void*)k_pcg_sweep<W, false> : (const void*)k_bicgstab_sweep<W, false>;
}

namespace {

// The division of a system whose rows have at most 6 entries on either side of
// the diagonal: rows of a block, as few blocks as hold them. False when the rows
// do not fit in the SMs' shared memory.
struct SweepDivision {
  int W, R, blocks, smem;
};
int divide_sweep(int n, int width, int bw, SweepDivision& v, bool& fits) {
  fits = false;
  if (width < 1 || width > 6) return 0;
  int dev = 0, sms = 0;
  MGPU_CUDA(cudaGetDevice(&dev));
  MGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MGPU_CUDA(cudaDeviceGetAttribute(&v.smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  v.W = width <= 3 ? 3 : width == 4 ? 4 : 6;
  const long room = v.smem - 2048 - sweep_smem(v.W, 0, bw);
  const int most = room > 0 ? (int)(room / sweep_row_bytes(v.W) / 32 * 32) : 0;
  // the polling threads keep their rows in a 32-bit mask; places are 16 bits
  if (most < 256 || bw > 32 * 32 * kPollWarps) return 0;
  const int blocks = (n + most - 1) / most;
  v.R = ((n + blocks - 1) / blocks + 31) / 32 * 32;
  v.blocks = (n + v.R - 1) / v.R;
  fits = blocks <= sms;
  return 0;
}

// The most rows that a level (rows ascending) has in one block: a thread a level and block.
__global__ void k_widest_level(int nlo, const int* __restrict__ lo_ptr, const int* __restrict__ lo_rows, int nup,
                               const int* __restrict__ up_ptr, const int* __restrict__ up_rows, int R, int blocks,
                               int* widest) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int mine = 0;
  if (t < (long)(nlo + nup) * blocks) {
    const int lev = (int)(t / blocks), blk = (int)(t % blocks);
    const int* ptr = lev < nlo ? lo_ptr + lev : up_ptr + (lev - nlo);
    const int* rows = lev < nlo ? lo_rows : up_rows;
    auto below = [&](long key) {
      int lo = ptr[0], hi = ptr[1];
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (rows[mid] < key)
          lo = mid + 1;
        else
          hi = mid;
      }
      return lo;
    };
    mine = below((blk + 1l) * R) - below((long)blk * R);
  }
  mine = __reduce_max_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine > 0) atomicMax(widest, mine);
}

}  // namespace

// Whether a system's sweeps are faster here than in krylov.cu (the caller then
// passes its width on in KrylovArgs, 0 otherwise). Each of the blocks polls bw
// values with the threads that no level needs, one after another, and a value
// waits half a round of them: blocks * bw / pollers against the levels, whose
// cost in krylov.cu is a grid-wide hop each. Measured on a B200 as krylov.cu's
// time over this one's, a BiCGStab+ILU(0) iteration (PCG+IC(0) gains more), by
// that quotient: channels of n = 65k, 100k, 126k, 151k, 180k, 216k rows in RCM
// order, at 1.8, 3.6, 5.3, 7.1, 9.3, 12: 2.5, 1.8, 1.4, 1.1, 0.98, 0.87; tetrahedra
// in natural order, 5.4 and 11: 1.4 and 0.98. Up to 8 it pays. Tetrahedra in RCM
// order, whose levels cross most blocks: 1.2 with 98 blocks (2.8), 0.97 with 129
// (4.0); narrow levels keep paying there: hexahedra in natural order, 130 blocks,
// at most 36 rows of a level in a block (5.4): 3.6. scratch: one int on the device;
// waits for stream s only where the answer depends on the widest level.
int plan_sweep(int n, int width, int bw, int nlo, const int* lo_ptr, const int* lo_rows, int nup, const int* up_ptr,
               const int* up_rows, int* scratch, cudaStream_t s, bool& pays) {
  constexpr long kRounds = 8;
  constexpr int kManyBlocks = 120, kNarrow = 64;
  SweepDivision v;
  if (int e = divide_sweep(n, width, bw, v, pays)) return e;
  if (!pays) return 0;
  const long polls = (long)v.blocks * bw, levels = std::min(nlo, nup);
  const int fewest = 32 * kPollWarps;
  if (v.blocks <= kManyBlocks && polls <= kRounds * fewest * levels) return 0;
  int widest = 0;
  const long threads = (long)(nlo + nup) * v.blocks;
  MGPU_CUDA(cudaMemsetAsync(scratch, 0, sizeof(int), s));
  k_widest_level<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(nlo, lo_ptr, lo_rows, nup, up_ptr, up_rows, v.R,
                                                                  v.blocks, scratch);
  MGPU_CUDA(cudaGetLastError());
  MGPU_CUDA(cudaMemcpyAsync(&widest, scratch, sizeof(int), cudaMemcpyDeviceToHost, s));
  MGPU_CUDA(cudaStreamSynchronize(s));
  const int pollers = std::max(kSweepThreads - (widest + 31) / 32 * 32, fewest);
  pays = polls <= kRounds * pollers * levels && (v.blocks <= kManyBlocks || widest <= kNarrow);
  return 0;
}

// The resident solve of a factored system that plan_sweep has found worth it,
// with the 6 n more work doubles that a.width > 0 stands for; *taken = false and
// no launch otherwise.
int launch_sweep(const KrylovArgs& a, bool pcg, cudaStream_t s, bool* taken) {
  *taken = false;
  SweepDivision v;
  bool fits = false;
  if (a.precond == 1) return 0;
  if (int e = divide_sweep(a.n, a.width, a.bw, v, fits)) return e;
  if (!fits) return 0;
  const int dyn = (int)sweep_smem(v.W, v.R, a.bw);
  const bool limits = g_spin_limit != 0u || g_exchange_limit != 0u;
  const void* fn = v.W == 3   ? sweep_kernel<3>(pcg, limits)
                   : v.W == 4 ? sweep_kernel<4>(pcg, limits)
                              : sweep_kernel<6>(pcg, limits);
  // the same limit on every call: another thread may be launching the kernel for another system
  MGPU_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem - 2048));
  KrylovArgs aa = a;
  int block = 0, RR = v.R, vgrid = krylov_grid(a.n, block, pcg ? 0 : 1);
  WaitLimits waits = wait_limits(g_spin_limit, g_exchange_limit);
  void* args[] = {&aa, &RR, &vgrid, &waits};
  MGPU_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned long long), s));
  MGPU_CUDA(cudaLaunchCooperativeKernel(fn, dim3(v.blocks), dim3(kSweepThreads), args, (size_t)dyn, s));
  *taken = true;
  return 0;
}

}  // namespace mgpu
