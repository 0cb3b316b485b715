// krylov_sweep.cu -- the FP64 parity form's ILU(0) / IC(0) solves on rows that
// stay in shared memory: cg_ic0 and PCG+ILU(0), bicgstab_ilu0
// (mod_uns_linsolver.f90:148-224, 405-461), with the row arithmetic and order of
// krylov.cu.
//
// What bounds these solves is the serial chain of the triangular sweeps: one hop
// per level, some 250 levels an iteration on a few thousand rows. In krylov.cu a
// hop is a chain of trips to L1 or L2: the row number, its pointers, its factor
// values, the neighbours' results, a block barrier or a poll of a value another
// block stores. Here a block owns a contiguous range of rows (as few blocks as
// shared memory allows: a hop inside a block is several times shorter than one
// between blocks), keeps their factor rows, level lists and the swept vector in
// shared memory, and a hop inside it is: shared-memory reads of the neighbours,
// the row's operations, a block barrier, with the next level's row already in
// registers. A value of another block is read from an exchange word
// (exchange.cuh) that the other block writes when it has the value. Rows are
// taken in level order on every block, so the least unfinished row can always
// proceed: the blocks are co-resident and a sweep ends. The sums take the
// layout-independent tree of exchange.cuh.

#include <algorithm>

#include "exchange.cuh"

namespace mgpu {
namespace {

constexpr int kSweepThreads = 512;

// A block's rows: sizes, and byte offsets into its shared memory. WO: most
// off-diagonal entries of a row.
template <int WO>
struct Sweep {
  int n, R, start, end, nsc;
  int wb, bw;        // first row of the column window; largest |column - row|
  int kind;          // 0 ILU(0), 2 IC(0)
  int cp, cps;       // chunk sums
  unsigned rseq;     // sums so far
  double* sums;      // super-chunk sums (2 halves x 2 sums x nsc)
  unsigned aseq;     // applications so far
  u64 *fwd, *bwd;    // exchange words (pairs) of the forward and backward results
  int w;             // double[R]: the swept vector
  int fd;            // double[R]: factor diagonal
  int fo;            // double[WO][R]: factor off-diagonals of a row, lower entries first, columns ascending
                     // (IC(0): the upper entries from the transposed factor)
  int ix;            // unsigned short[WO][R]: their columns, from wb
  int meta;          // unsigned short[R]: lower entries | upper entries << 4
  int olo, oup;      // unsigned short[R]: rows in lower / upper level order
  int plo, pup;      // unsigned short[R + 1]: first of each local level
  int nlo, nup;      // local levels (those with a row of this block)
};

constexpr int sweep_row_bytes(int WO) { return 16 + 10 * WO + 2 * 5; }
inline int sweep_smem(int WO, int R, int cps) { return sweep_row_bytes(WO) * R + 16 + 16 * cps; }

template <int WO>
__device__ __forceinline__ void sweep_views(Sweep<WO>& S, int R, int cps) {
  S.R = R;
  S.cps = cps;
  S.cp = 0;
  S.w = 16 * cps;
  S.fd = S.w + 8 * R;
  S.fo = S.fd + 8 * R;
  S.ix = S.fo + 8 * WO * R;
  S.meta = S.ix + 2 * WO * R;
  S.olo = S.meta + 2 * R;
  S.oup = S.olo + 2 * R;
  S.plo = S.oup + 2 * R;
  S.pup = S.plo + 2 * (R + 1);
}

// The block's rows of a level order (ptr, rows: the system's, rows ascending in
// a level) as local lists; returns the number of local levels. scratch: int[2 * R]
// in shared memory.
__device__ __forceinline__ int local_levels(const int* __restrict__ ptr, const int* __restrict__ rows, int nlev,
                                            int start, int end, int out, int lptr, int scratch) {
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
  __syncthreads();
  return nl;
}

// The block's part of the system in shared memory, its words cleared; the
// barrier puts every block's clears (and zeroed x) before what follows.
template <int WO, int K>
__device__ __forceinline__ bool sweep_prologue(const KrylovArgs& a, VGrid& g, Sweep<WO>& S) {
  const int T = blockDim.x, tid = threadIdx.x;
  S.wb = max(0, S.start - S.bw);
  S.nlo = local_levels(a.lo_ptr, a.lo_rows, a.nlev_lo, S.start, S.end, S.olo, S.plo, S.fo);
  S.nup = local_levels(a.up_ptr, a.up_rows, a.nlev_up, S.start, S.end, S.oup, S.pup, S.fo);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int l = k * T + tid, i = S.start + l;
    if (i >= S.end) continue;
    const int rb = a.row_ptr[i], re = a.row_ptr[i + 1], di = a.diag[i];
    const int nl = di - rb;
#pragma unroll
    for (int t = 0; t < WO; ++t)
      if (rb + t + (t >= nl) < re) {
        const int e = rb + t + (t >= nl);  // the diagonal is skipped
        smem_at<double>(S.fo, t * S.R + l) = a.fval[S.kind == 2 && t >= nl ? a.lt_pos[e] : e];
        smem_at<unsigned short>(S.ix, t * S.R + l) = (unsigned short)(a.col[e] - S.wb);
      }
    smem_at<double>(S.fd, l) = a.fval[di];
    smem_at<unsigned short>(S.meta, l) = (unsigned short)(nl | (re - di - 1) << 4);
    S.fwd[2l * i] = S.fwd[2l * i + 1] = 0ull;
    S.bwd[2l * i] = S.bwd[2l * i + 1] = 0ull;
    if (a.zero_x) a.x[i] = 0.0;
  }
  return vg_sync(g, a.st);
}

// A row of the next level, read ahead of the barrier before it.
template <int WO>
struct Fetched {
  int l;  // local row (-1: none)
  int m;  // entries to apply
  double f[WO];
  int c[WO];  // their columns, from the block's first row
  double fd;
};

template <int WO, bool FWD>
__device__ __forceinline__ void fetch_row(const Sweep<WO>& S, int idx, int e, Fetched<WO>& r) {
  r.l = -1;
  if (idx >= e) return;
  const int l = smem_at<unsigned short>(FWD ? S.olo : S.oup, idx);
  const unsigned meta = smem_at<unsigned short>(S.meta, l);
  const int nl = meta & 15u, nu = meta >> 4, off = S.wb - S.start;
  r.l = l;
  r.m = FWD ? nl : nu;
  r.fd = smem_at<double>(S.fd, l);
#pragma unroll
  for (int t = 0; t < WO; ++t)
    if (t < r.m) {
      // IC(0)'s backward sweep applies the entries in descending column order
      const int p = FWD ? t : (S.kind == 2 ? nl + nu - 1 - t : nl + t);
      r.f[t] = smem_at<double>(S.fo, p * S.R + l);
      r.c[t] = (int)smem_at<unsigned short>(S.ix, p * S.R + l) + off;
    }
}

template <int WO, bool FWD>
__device__ __forceinline__ bool sweep_row(const Sweep<WO>& S, const Fetched<WO>& r, DevStatus* st) {
  const u64* words = FWD ? S.fwd : S.bwd;
  double v[WO];
  bool ok = true;
#pragma unroll
  for (int t = 0; t < WO; ++t)
    if (t < r.m) {
      if ((unsigned)r.c[t] < (unsigned)S.R) {
        v[t] = smem_at<double>(S.w, r.c[t]);
      } else {
        const u64* p = words + 2l * (S.start + r.c[t]);
        u64 lo, hi;
        ld_pair(p, lo, hi);
        unsigned spins = 0;
        while (((unsigned)(lo >> 32) != S.aseq || (unsigned)(hi >> 32) != S.aseq) && ok) {
          ok = keep_polling(spins, st);
          ld_pair(p, lo, hi);
        }
        v[t] = __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
      }
    }
  double s = smem_at<double>(S.w, r.l);
#pragma unroll
  for (int t = 0; t < WO; ++t)
    if (t < r.m) s = s - r.f[t] * v[t];
  if (!FWD || S.kind == 2) s = s / r.fd;
  smem_at<double>(S.w, r.l) = s;
  // rows within a bandwidth of the range's end (forward) or start (backward)
  // may be another block's neighbours
  const bool out = FWD ? r.l + S.bw >= S.end - S.start && S.end < S.n : r.l < S.bw && S.start > 0;
  if (out) st_pair(const_cast<u64*>(words) + 2l * (S.start + r.l), s, S.aseq);
  return ok;
}

template <int WO, bool FWD>
__device__ __forceinline__ bool sweep_half(const Sweep<WO>& S, DevStatus* st) {
  const int tid = threadIdx.x, T = blockDim.x;
  const int nlev = FWD ? S.nlo : S.nup, ptr = FWD ? S.plo : S.pup;
  bool ok = true;
  Fetched<WO> r;
  int e = smem_at<unsigned short>(ptr, 1);
  fetch_row<WO, FWD>(S, smem_at<unsigned short>(ptr, 0) + tid, e, r);
  for (int lev = 0; lev < nlev; ++lev) {
    if (r.l >= 0) ok = sweep_row<WO, FWD>(S, r, st) && ok;
    for (int idx = smem_at<unsigned short>(ptr, lev) + T + tid; idx < e; idx += T) {
      fetch_row<WO, FWD>(S, idx, e, r);
      ok = sweep_row<WO, FWD>(S, r, st) && ok;
    }
    r.l = -1;
    if (lev + 1 < nlev) {
      const int b = e;
      e = smem_at<unsigned short>(ptr, lev + 2);
      fetch_row<WO, FWD>(S, b + tid, e, r);
    }
    __syncthreads();
  }
  return ok;
}

// z = M^-1 src for the block's rows (z[k] of this thread's row in tile k). The
// words of an application are written again only after a sum over all blocks,
// which each block joins when it has read all it needs.
template <int WO, int K>
__device__ __forceinline__ bool sweep_apply(Sweep<WO>& S, const double (&src)[K], double (&z)[K], DevStatus* st) {
  const int T = blockDim.x, tid = threadIdx.x;
  ++S.aseq;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int l = k * T + tid;
    if (S.start + l < S.end) smem_at<double>(S.w, l) = src[k];
  }
  __syncthreads();
  bool ok = sweep_half<WO, true>(S, st);
  ok = sweep_half<WO, false>(S, st) && ok;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int l = k * T + tid;
    z[k] = S.start + l < S.end ? smem_at<double>(S.w, l) : 0.0;
  }
  return __syncthreads_and(ok) != 0;
}

// y_i = A_i . x in csr_matvec order
__device__ __forceinline__ double row_product(const KrylovArgs& a, const double* x, int i) {
  const int b = a.row_ptr[i], e = a.row_ptr[i + 1];
  double v[8], xv[8];
#pragma unroll
  for (int t = 0; t < 8; ++t)
    if (b + t < e) {
      v[t] = a.aval[b + t];
      xv[t] = ldv(&x[a.col[b + t]]);
    }
  double y = 0.0;
#pragma unroll
  for (int t = 0; t < 8; ++t)
    if (b + t < e) y = y + v[t] * xv[t];
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

template <int WO, int K>
__device__ __forceinline__ void sweep_begin(const KrylovArgs& a, const VGrid& g, Sweep<WO>& S, int R, int bw) {
  S.n = a.n;
  S.bw = bw;
  S.kind = a.precond;
  S.start = g.rank * R;
  S.end = min(a.n, S.start + R);
  S.nsc = (a.n + kSuperRows - 1) / kSuperRows;
  S.rseq = S.aseq = 0u;
  S.sums = a.z;
  sweep_views<WO>(S, R, K * (blockDim.x / 32));
}

// the rows of this thread: f(tile k, row i)
#define MGPU_OWN_ROWS(k, i)                                        \
  _Pragma("unroll") for (int k = 0; k < K; ++k)                    \
    if (const int i = S.start + k * (int)blockDim.x + (int)threadIdx.x; i < S.end)

// sum over all rows of the per-row values c0[k] (c1[k]) into out
template <int K, typename State>
__device__ __forceinline__ bool sum1(State& S, VGrid& g, DevStatus* st, const double (&c0)[K], double& out) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double c[1] = {c0[k]};
    resident_put<1>(S.cp, S.cps, k, c);
  }
  double t[1];
  if (!resident_total<1>(S, g, st, t)) return false;
  out = t[0];
  return true;
}
template <int K, typename State>
__device__ __forceinline__ bool sum2(State& S, VGrid& g, DevStatus* st, const double (&c0)[K], const double (&c1)[K],
                                     double (&out)[2]) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double c[2] = {c0[k], c1[k]};
    resident_put<2>(S.cp, S.cps, k, c);
  }
  return resident_total<2>(S, g, st, out);
}

// k_pcg (krylov.cu) with ILU(0) or IC(0)
template <int WO, int K>
__global__ void __launch_bounds__(kSweepThreads, 1) k_pcg_sweep(KrylovArgs a, int R, int bw) {
  if (a.st->abort) return;
  VGrid g = whole_grid(a.bar, a.partials, true);
  Sweep<WO> S;
  sweep_begin<WO, K>(a, g, S, R, bw);
  S.fwd = reinterpret_cast<u64*>(a.s);   // s, t
  S.bwd = reinterpret_cast<u64*>(a.ph);  // ph, sh
  double* x = a.x;
  double* p = a.p;
  double r[K], z[K], q[K], pk[K], c[K];
  if (!sweep_prologue<WO, K>(a, g, S)) return;
#pragma unroll
  for (int k = 0; k < K; ++k) r[k] = z[k] = q[k] = pk[k] = c[k] = 0.0;
  MGPU_OWN_ROWS(k, i) c[k] = a.b[i] * a.b[i];
  double bb;
  if (!sum1<K>(S, g, a.st, c, bb)) return;
  const double bnrm = sqrt(bb);
  if (bnrm == 0.0) {
    MGPU_OWN_ROWS(k, i) x[i] = 0.0;
    sweep_result(a, 0, 0.0, 0);
    return;
  }
  if (*a.ferr != 0) {
    sweep_result(a, 0, 0.0, *a.ferr + 10);
    return;
  }
  MGPU_OWN_ROWS(k, i) {
    r[k] = a.b[i] - row_product(a, x, i);
    c[k] = r[k] * r[k];
  }
  double rr;
  if (!sum1<K>(S, g, a.st, c, rr)) return;
  double res = sqrt(rr) / bnrm;
  if (res <= a.tol) {
    sweep_result(a, 0, res, 0);
    return;
  }
  double rz;
  if (!sweep_apply<WO, K>(S, r, z, a.st)) return;
#pragma unroll
  for (int k = 0; k < K; ++k) c[k] = r[k] * z[k];
  MGPU_OWN_ROWS(k, i) {
    pk[k] = z[k];
    p[i] = pk[k];
  }
  if (!sum1<K>(S, g, a.st, c, rz)) return;  // its barrier shows every block's p
  int ierr = 0, it;
  for (it = 1; it <= a.maxit; ++it) {
    MGPU_OWN_ROWS(k, i) {
      q[k] = row_product(a, p, i);
      c[k] = pk[k] * q[k];
    }
    double pap;
    if (!sum1<K>(S, g, a.st, c, pap)) return;
    if (fabs(pap) < DTINY) {
      ierr = 2;
      break;
    }
    const double alpha = rz / pap;
    MGPU_OWN_ROWS(k, i) {
      x[i] = x[i] + alpha * pk[k];
      r[k] = r[k] - alpha * q[k];
      c[k] = r[k] * r[k];
    }
    if (!sum1<K>(S, g, a.st, c, rr)) return;
    res = sqrt(rr) / bnrm;
    if (res <= a.tol) {
      sweep_result(a, it, res, 0);
      return;
    }
    double rz_new;
    if (!sweep_apply<WO, K>(S, r, z, a.st)) return;
#pragma unroll
    for (int k = 0; k < K; ++k) c[k] = r[k] * z[k];
    if (!sum1<K>(S, g, a.st, c, rz_new)) return;
    if (fabs(rz) < DTINY) {
      ierr = 2;
      break;
    }
    const double beta = rz_new / rz;
    MGPU_OWN_ROWS(k, i) {
      pk[k] = z[k] + beta * pk[k];
      p[i] = pk[k];
    }
    if (!vg_sync(g, a.st)) return;
    rz = rz_new;
  }
  if (ierr == 0) ierr = 1;
  sweep_result(a, it, res, ierr);
}

// k_bicgstab (krylov.cu) with ILU(0)
template <int WO, int K>
__global__ void __launch_bounds__(kSweepThreads, 1) k_bicgstab_sweep(KrylovArgs a, int R, int bw) {
  if (a.st->abort) return;
  VGrid g = whole_grid(a.bar, a.partials, true);
  Sweep<WO> S;
  sweep_begin<WO, K>(a, g, S, R, bw);
  S.fwd = reinterpret_cast<u64*>(a.p);  // p, v
  S.bwd = reinterpret_cast<u64*>(a.s);  // s, t
  double* x = a.x;
  double *r0 = a.r0, *ph = a.ph, *sh = a.sh;
  double r[K], p[K], v[K], y[K], z[K], t[K], c[K], e[K];
  if (!sweep_prologue<WO, K>(a, g, S)) return;
#pragma unroll
  for (int k = 0; k < K; ++k) r[k] = p[k] = v[k] = y[k] = z[k] = t[k] = c[k] = e[k] = 0.0;
  MGPU_OWN_ROWS(k, i) c[k] = a.b[i] * a.b[i];
  double bb;
  if (!sum1<K>(S, g, a.st, c, bb)) return;
  const double bnrm = sqrt(bb);
  if (bnrm == 0.0) {
    MGPU_OWN_ROWS(k, i) x[i] = 0.0;
    sweep_result(a, 0, 0.0, 0);
    return;
  }
  if (*a.ferr != 0) {
    sweep_result(a, 0, 0.0, *a.ferr + 10);
    return;
  }
  MGPU_OWN_ROWS(k, i) {
    r[k] = a.b[i] - row_product(a, x, i);
    r0[i] = r[k];
    c[k] = r[k] * r[k];
  }
  double rho_next;
  if (!sum1<K>(S, g, a.st, c, rho_next)) return;
  double res = sqrt(rho_next) / bnrm;
  if (res <= a.tol) {
    sweep_result(a, 0, res, 0);
    return;
  }
  double rho_old = 1.0, alpha = 1.0, omega = 1.0;
  int ierr = 0, it;
  for (it = 1; it <= a.maxit; ++it) {
    const double rho = rho_next;
    if (fabs(rho) < DTINY) {
      ierr = 2;
      break;
    }
    const double beta = (rho / rho_old) * (alpha / omega);
#pragma unroll
    for (int k = 0; k < K; ++k) p[k] = r[k] + beta * (p[k] - omega * v[k]);
    if (!sweep_apply<WO, K>(S, p, y, a.st)) return;
    MGPU_OWN_ROWS(k, i) ph[i] = y[k];
    if (!vg_sync(g, a.st)) return;
    MGPU_OWN_ROWS(k, i) {
      v[k] = row_product(a, ph, i);
      c[k] = r0[i] * v[k];
    }
    double d1;
    if (!sum1<K>(S, g, a.st, c, d1)) return;
    alpha = rho / d1;
    // r becomes s
#pragma unroll
    for (int k = 0; k < K; ++k) {
      r[k] = r[k] - alpha * v[k];
      c[k] = r[k] * r[k];
    }
    double d2;
    if (!sum1<K>(S, g, a.st, c, d2)) return;
    const double snrm = sqrt(d2);
    if (snrm / bnrm <= a.tol) {
      MGPU_OWN_ROWS(k, i) x[i] = x[i] + alpha * y[k];
      sweep_result(a, it, snrm / bnrm, 0);
      return;
    }
    if (!sweep_apply<WO, K>(S, r, z, a.st)) return;
    MGPU_OWN_ROWS(k, i) sh[i] = z[k];
    if (!vg_sync(g, a.st)) return;
    MGPU_OWN_ROWS(k, i) {
      t[k] = row_product(a, sh, i);
      c[k] = t[k] * t[k];
      e[k] = t[k] * r[k];
    }
    double d3[2];
    if (!sum2<K>(S, g, a.st, c, e, d3)) return;
    const double tt = d3[0];
    if (tt < DTINY) {
      ierr = 2;
      break;
    }
    omega = d3[1] / tt;
    if (fabs(omega) < DTINY) {
      ierr = 2;
      break;
    }
    MGPU_OWN_ROWS(k, i) {
      x[i] = x[i] + alpha * y[k] + omega * z[k];
      r[k] = r[k] - omega * t[k];
      c[k] = r[k] * r[k];
      e[k] = r[k] * r0[i];
    }
    double d4[2];
    if (!sum2<K>(S, g, a.st, c, e, d4)) return;
    res = sqrt(d4[0]) / bnrm;
    if (res <= a.tol) {
      sweep_result(a, it, res, 0);
      return;
    }
    rho_next = d4[1];
    rho_old = rho;
  }
  if (ierr == 0) {
    ierr = 1;
    it = a.maxit;
  }
  sweep_result(a, it, res, ierr);
}
#undef MGPU_OWN_ROWS

template <int WO>
const void* sweep_kernel(int K, bool pcg) {
  switch (K) {
    case 1: return pcg ? (const void*)k_pcg_sweep<WO, 1> : (const void*)k_bicgstab_sweep<WO, 1>;
    case 2: return pcg ? (const void*)k_pcg_sweep<WO, 2> : (const void*)k_bicgstab_sweep<WO, 2>;
    case 4: return pcg ? (const void*)k_pcg_sweep<WO, 4> : (const void*)k_bicgstab_sweep<WO, 4>;
    default: return pcg ? (const void*)k_pcg_sweep<WO, 6> : (const void*)k_bicgstab_sweep<WO, 6>;
  }
}

}  // namespace

// The resident solve of a factored system whose rows have at most 7 entries and
// fit in the SMs' shared memory, column windows in 16 bits; *taken = false and
// no launch otherwise.
int launch_sweep(const KrylovArgs& a, bool pcg, cudaStream_t s, bool* taken) {
  *taken = false;
  if (a.precond == 1 || a.width < 1 || a.width > 7 || a.n < 64) return 0;
  int dev = 0, sms = 0, smem = 0;
  MGPU_CUDA(cudaGetDevice(&dev));
  MGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MGPU_CUDA(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const int WO = a.width <= 5 ? 4 : 6;
  const int room = smem - 2048 - sweep_smem(WO, 0, 6 * (kSweepThreads / 32));
  const int most = std::min(room / sweep_row_bytes(WO) / kSuperRows * kSuperRows, 6 * kSweepThreads);
  const int blocks = (a.n + most - 1) / most;
  const int R = ((a.n + blocks - 1) / blocks + kSuperRows - 1) / kSuperRows * kSuperRows;
  const int grid = (a.n + R - 1) / R;
  if (grid > sms || a.n > 10 * 256 * kSuperRows || R + 2l * a.bw > 65535) return 0;
  int K = (R + kSweepThreads - 1) / kSweepThreads;
  K = K <= 2 ? K : K <= 4 ? 4 : 6;
  const int dyn = sweep_smem(WO, R, K * (kSweepThreads / 32));
  const void* fn = WO == 4 ? sweep_kernel<4>(K, pcg) : sweep_kernel<6>(K, pcg);
  MGPU_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn));
  KrylovArgs aa = a;
  int RR = R, bw = a.bw;
  void* args[] = {&aa, &RR, &bw};
  MGPU_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned long long), s));
  MGPU_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kSweepThreads), args, (size_t)dyn, s));
  *taken = true;
  return 0;
}

}  // namespace mgpu
