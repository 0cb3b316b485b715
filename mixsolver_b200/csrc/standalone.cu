// standalone.cu -- C-ABI entry points that work on plain host arrays:
// Krylov solves and SpMV on a CSR matrix (the mod_uns_linsolver interface),
// and the mesh pipeline (connectivity, geometry, RCM ordering).

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "assembly.cuh"
#include "case.cuh"
#include "device_topo.h"
#include "mesh_host.h"

namespace mgpu {
extern unsigned g_spin_limit;  // krylov.cu: the spin_limit tuning key
extern unsigned g_poll_ns;     // krylov.cu: the barrier_poll_ns tuning key
extern int g_cheb_degree;      // the cheb_degree and cheb_ratio tuning keys
extern double g_cheb_ratio;
void cheb_params(long n, int& k, double& ratio);  // krylov.cu
extern int g_prefetch_mb;      // l2_prefetch_mb
size_t page_floats(int n, int W, const ResidentPlan& plan);  // krylov_resident.cu
int plan_sweep(int n, int width, int bw, int nlo, const int* lo_ptr, const int* lo_rows, int nup, const int* up_ptr,
               const int* up_rows, int* scratch, cudaStream_t s, bool& pays);  // krylov_sweep.cu
}

using namespace mgpu;

namespace {

// Device buffers of one call: pieces of one allocation of the size that the
// caller reserved (an allocation and a release for each buffer took most of a
// small solve's time), anything beyond it on its own.
struct DevBuf {
  std::vector<void*> p;
  char* base = nullptr;
  size_t left = 0;
  ~DevBuf() {
    for (void* q : p) cudaFree(q);
  }
  int reserve(size_t bytes) {
    void* q = nullptr;
    MGPU_CUDA(cudaMalloc(&q, bytes));
    p.push_back(q);
    base = (char*)q;
    left = bytes;
    return 0;
  }
  template <typename T>
  int alloc(T*& out, size_t n) {
    const size_t bytes = (std::max<size_t>(n, 1) * sizeof(T) + 255) / 256 * 256;
    if (bytes <= left) {
      out = (T*)base;
      base += bytes;
      left -= bytes;
      return 0;
    }
    void* q = nullptr;
    MGPU_CUDA(cudaMalloc(&q, bytes));
    p.push_back(q);
    out = (T*)q;
    return 0;
  }
  template <typename T>
  int up(T*& out, const T* h, size_t n) {
    if (int e = alloc(out, n)) return e;
    if (n) MGPU_CUDA(cudaMemcpy(out, h, n * sizeof(T), cudaMemcpyHostToDevice));
    return 0;
  }
};

#define TRY(x)                 \
  do {                         \
    int rc_ = (x);             \
    if (rc_ != 0) return rc_;  \
  } while (0)

// What the solves need of a host CSR pattern (1-based, columns ascending).
struct Pattern {
  int *rp = nullptr, *col = nullptr, *diag = nullptr, *mirror = nullptr;  // 0-based, on the device
  int nnz = 0;
  bool symmetric = false, full_diag = false;
  // most entries of a row on one side of the diagonal (0: some row's columns do not ascend, and its entries
  // before and after the diagonal need not be those of smaller and larger columns), largest |column - row|
  int width = 0, bw = 0;
};

enum { kNoDiag, kUnpaired, kUnsorted, kSide, kFar, kBadColumn, kFlags };

// The 0-based pattern, the diagonal's and the transposed entries' positions;
// flags: rows without a diagonal entry, entries without a transposed one, rows
// whose columns do not ascend, the most entries on one side of a diagonal, the
// largest |column - row|, columns out of range. A search ends at the first
// larger column, so an entry after one is not found. A thread a row: the
// searches run along rows of a few entries (on the host they took longer than
// the solve).
__global__ void k_csr_pattern(int n, const int* __restrict__ rp1, const int* __restrict__ col1, int* rp, int* col,
                              int* diag, int* mirror, int* flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  rp[i] = rp1[i] - 1;
  if (i == n) return;
  const int b = rp1[i] - 1, e = rp1[i + 1] - 1;
  int d = -1, lower = 0, upper = 0, far = 0, prev = -1;
  bool past = false, sorted = true;  // past: a column after the diagonal has been met
  for (int k = b; k < e; ++k) {
    const int j = col1[k] - 1;
    col[k] = j;
    if (j < 0 || j >= n) {
      atomicOr(&flags[kBadColumn], 1);
      continue;
    }
    far = max(far, abs(j - i));
    lower += j < i;
    upper += j > i;
    if (j == i && d < 0 && !past) d = k;
    past = past || j > i;
    sorted = sorted && j > prev;
    prev = j;
    int m = -1;
    for (int q = rp1[j] - 1, qe = rp1[j + 1] - 1; q < qe; ++q) {
      const int c = col1[q] - 1;
      if (c == i) m = q;
      if (c >= i) break;
    }
    if (m < 0) {
      atomicOr(&flags[kUnpaired], 1);
      m = k;
    }
    mirror[k] = m;
  }
  diag[i] = d;
  if (d < 0) atomicOr(&flags[kNoDiag], 1);
  if (!sorted) atomicOr(&flags[kUnsorted], 1);
  atomicMax(&flags[kSide], max(lower, upper));
  atomicMax(&flags[kFar], far);
}

// Every row's entries lie within the arrays (the device reads them unchecked).
int check_rows(int n, const int32_t* row_ptr) {
  const int end = row_ptr[n];
  int bad = end < 1;
  for (int i = 0; i <= n; ++i) bad |= (row_ptr[i] < 1) | (row_ptr[i] > end);  // no early exit: it vectorises
  if (bad) set_error("CSR matrix: a row pointer out of range");
  return bad ? MGPU_E_ARG : 0;
}

int load_pattern(int n, const int32_t* row_ptr, const int32_t* col_idx, DevBuf& B, Pattern& P) {
  P.nnz = row_ptr[n] - 1;
  int *rp1, *col1, *flags;
  TRY(B.up(rp1, row_ptr, n + 1));
  TRY(B.up(col1, col_idx, P.nnz));
  TRY(B.alloc(P.rp, n + 1));
  TRY(B.alloc(P.col, P.nnz));
  TRY(B.alloc(P.diag, n));
  TRY(B.alloc(P.mirror, P.nnz));
  TRY(B.alloc(flags, kFlags));
  MGPU_CUDA(cudaMemset(flags, 0, kFlags * sizeof(int)));
  k_csr_pattern<<<ceil_div(n + 1, 128), 128>>>(n, rp1, col1, P.rp, P.col, P.diag, P.mirror, flags);
  MGPU_LAUNCH_CHECK("k_csr_pattern");
  int h[kFlags];
  MGPU_CUDA(cudaMemcpy(h, flags, sizeof(h), cudaMemcpyDeviceToHost));
  if (h[kBadColumn]) {
    set_error("CSR matrix: a column out of range");
    return MGPU_E_ARG;
  }
  P.full_diag = !h[kNoDiag];
  P.symmetric = !h[kUnpaired];
  P.width = h[kUnsorted] ? 0 : std::max(h[kSide], 1);
  P.bw = h[kFar];
  return 0;
}

// The triangular level sets (rows by level, ascending in a level); each row has
// its diagonal entry before any larger column.
struct Levels {
  std::vector<int> lo_ptr, lo_rows, up_ptr, up_rows;
  int nlo = 0, nup = 0;
};

void level_sets(int n, const int32_t* rp, const int32_t* col, Levels& L) {
  std::vector<int> lev(n, 0);
  auto bucket = [&](int nl, std::vector<int>& ptr, std::vector<int>& rows) {
    ptr.assign(nl + 1, 0);
    for (int i = 0; i < n; ++i) ptr[lev[i] + 1]++;
    for (int l = 0; l < nl; ++l) ptr[l + 1] += ptr[l];
    rows.assign(n, 0);
    std::vector<int> f(ptr.begin(), ptr.end() - 1);
    for (int i = 0; i < n; ++i) rows[f[lev[i]]++] = i;
  };
  for (int i = 0; i < n; ++i) {
    int l = 0;
    for (int k = rp[i] - 1; col[k] - 1 < i; ++k) l = std::max(l, lev[col[k] - 1] + 1);
    lev[i] = l;
    L.nlo = std::max(L.nlo, l + 1);
  }
  bucket(L.nlo, L.lo_ptr, L.lo_rows);
  for (int i = n - 1; i >= 0; --i) {
    int l = 0, k = rp[i] - 1;
    while (col[k] - 1 != i) ++k;
    for (++k; k < rp[i + 1] - 1; ++k) l = std::max(l, lev[col[k] - 1] + 1);
    lev[i] = l;
    L.nup = std::max(L.nup, l + 1);
  }
  bucket(L.nup, L.up_ptr, L.up_rows);
}

// The pressure solver of the mixed and FP64 polynomial forms on a host CSR
// system: the case's own kernels (k_pcg_mixed / k_pcg_poly64) with the
// arguments a case would give them, the ELL copy built on the device.
template <typename V>
int poly_solve(int n, const Pattern& P, DevBuf& B, const double* val, const double* b, double* x, double tol, int maxit,
                      int cheb_degree, double cheb_ratio, int* it, double* res, int* ierr) {
  const int nnz = P.nnz;
  int *drp = P.rp, *dcol = P.col, *ddiag = P.diag, *dferr;
  double *dval, *db, *dx, *dkw, *dpart, *dred;
  V *da, *ddinv, *dw;
  unsigned long long* dbar;
  DevStatus* dst;
  MgpuIterRec* drec;
  TRY(B.up(dval, val, nnz));
  TRY(B.up(db, b, n));
  TRY(B.up(dx, x, n));
  TRY(B.alloc(dkw, 10 * (size_t)n));
  TRY(B.alloc(dpart, 4 * 4096));
  TRY(B.alloc(dred, (size_t)mixed_red_words(n)));
  TRY(B.alloc(ddinv, n));
  TRY(B.alloc(dw, 10 * (size_t)n));
  TRY(B.alloc(dbar, 1));
  TRY(B.alloc(dferr, 1));
  TRY(B.alloc(dst, 1));
  TRY(B.alloc(drec, 1));
  int W = 0, *ell = nullptr;
  long ld = 0;
  TopoAlloc alloc = [&](int*& q, size_t k) { return B.alloc(q, k); };
  int bw = -1;  // the resident solve exchanges between blocks both ways: symmetric patterns only
  TRY(device_ell(n, drp, dcol, 8, W, ld, ell, alloc, 0, &bw));
  ResidentPlan plan;
  if (sizeof(V) == 4 && P.symmetric) TRY(plan_resident(n, W, (int)ld, ell, bw, plan, dferr, 0));
  TRY(B.alloc(da, nnz + page_floats(n, W, plan)));
  V* dev = nullptr;
  double* dev64 = nullptr;  // the mixed form's FP64 conjugate-gradient product
  if (ell) {
    TRY(B.alloc(dev, (size_t)W * ld));
    MGPU_CUDA(cudaMemset(dev, 0, sizeof(V) * (size_t)W * ld));
    if (sizeof(V) == 4) {
      TRY(B.alloc(dev64, (size_t)W * ld));
      MGPU_CUDA(cudaMemset(dev64, 0, sizeof(double) * (size_t)W * ld));
    }
  }
  DevStatus h{};
  h.nan_key = ~0ull;
  h.spin_limit = g_spin_limit;
  h.poll_ns = g_poll_ns;
  MGPU_CUDA(cudaMemcpy(dst, &h, sizeof(h), cudaMemcpyHostToDevice));
  MGPU_CUDA(cudaMemset(drec, 0, sizeof(MgpuIterRec)));
  KrylovArgs a{};
  a.n = n;
  a.row_ptr = drp;
  a.col = dcol;
  a.diag = ddiag;
  a.aval = dval;
  a.b = db;
  a.x = dx;
  a.r = dkw;
  a.p = dkw + 2l * n;
  a.v = dkw + 3l * n;
  a.s = dkw + 4l * n;
  a.tol = tol;
  a.maxit = maxit;
  a.precond = 1;
  a.partials = dpart;
  a.bar = dbar;
  a.st = dst;
  a.recs = drec;
  a.ferr = dferr;
  const bool mixed = sizeof(V) == 4;
  const double row_bytes = mixed ? mixed_row_bytes(W) : 16.0 * W + 80.0;
  const bool big = (double)n * row_bytes > g_prefetch_mb * 1048576.0;
  MixedArgsT<V> m{da,   ddinv, dw, 1e-4, cheb_degree, cheb_ratio, W, ell, dev, dred, (ell && big) ? 1 : 0, 0.0,
                  (int)ld, 0,  dev64, plan};
  if constexpr (sizeof(V) == 4)
    TRY(launch_pcg_mixed(a, m, 0));
  else
    TRY(launch_pcg_poly64(a, m, 0));
  MGPU_CUDA(cudaDeviceSynchronize());
  MgpuIterRec r{};
  MGPU_CUDA(cudaMemcpy(&r, drec, sizeof(r), cudaMemcpyDeviceToHost));
  MGPU_CUDA(cudaMemcpy(&h, dst, sizeof(h), cudaMemcpyDeviceToHost));
  MGPU_CUDA(cudaMemcpy(x, dx, sizeof(double) * n, cudaMemcpyDeviceToHost));
  if (h.timeout) {
    set_error("a bounded device wait ran out (grid barrier)");
    return MGPU_E_TIMEOUT;
  }
  *it = r.lin_it[0];
  *res = r.lin_res[0];
  *ierr = r.lin_ierr[0];
  return 0;
}

}  // namespace

extern "C" {

int mgpu_krylov_solve(int n, const int32_t* row_ptr, const int32_t* col_idx, const double* val, const double* b,
                      double* x, double tol, int maxit, int method, int norm_mode, int* it, double* res,
                      int* ierr) {
  if (n <= 0 || !row_ptr || !col_idx || !val || !b || !x || !it || !res || !ierr || method < 0 || method > 4 ||
      maxit < 0) {
    set_error("mgpu_krylov_solve: invalid argument");
    return MGPU_E_ARG;
  }
  TRY(check_rows(n, row_ptr));
  DevBuf B;
  const size_t nz = row_ptr[n] - 1;
  TRY(B.reserve(40 * nz + 220 * (size_t)n + (1 << 18)));
  Pattern P;
  TRY(load_pattern(n, row_ptr, col_idx, B, P));
  const int precond = (method == 0 || method == 4) ? 0 : (method == 2 ? 2 : 1);
  const bool bicg = method == 0 || method == 3;
  *it = 0;
  *res = 0.0;
  *ierr = 0;
  if (!P.full_diag) {
    // the reference checks b = 0 first, then the missing diagonal
    bool bz = true;
    for (int i = 0; i < n; ++i) bz = bz && (b[i] == 0.0);
    if (bz) {
      for (int i = 0; i < n; ++i) x[i] = 0.0;
      return 0;
    }
    *ierr = (precond == 1) ? (bicg ? 12 : 2) : 11;
    return 0;
  }
  if (precond == 2 && !P.symmetric) {
    set_error("mgpu_krylov_solve: IC(0) needs a structurally symmetric pattern");
    return MGPU_E_ARG;
  }
  Levels L;
  if (precond != 1) level_sets(n, row_ptr, col_idx, L);
  const int nnz = P.nnz;
  int *drp = P.rp, *dcol = P.col, *ddiag = P.diag, *dmir = P.mirror, *dlop, *dlor, *dupp, *dupr, *dferr;
  double *dval, *dfval, *db, *dx, *dkw, *dpart;
  unsigned long long* dbar;
  DevStatus* dst;
  MgpuIterRec* drec;
  TRY(B.up(dlop, L.lo_ptr.data(), L.lo_ptr.size()));
  TRY(B.up(dlor, L.lo_rows.data(), L.lo_rows.size()));
  TRY(B.up(dupp, L.up_ptr.data(), L.up_ptr.size()));
  TRY(B.up(dupr, L.up_rows.data(), L.up_rows.size()));
  TRY(B.up(dval, val, nnz));
  TRY(B.alloc(dfval, nnz));
  TRY(B.up(db, b, n));
  TRY(B.up(dx, x, n));
  TRY(B.alloc(dkw, 16 * (size_t)n));
  TRY(B.alloc(dpart, 4 * 4096));
  TRY(B.alloc(dbar, 1));
  TRY(B.alloc(dferr, 1));
  TRY(B.alloc(dst, 1));
  TRY(B.alloc(drec, 1));
  DevStatus h{};
  h.nan_key = ~0ull;
  h.spin_limit = g_spin_limit;
  h.poll_ns = g_poll_ns;
  MGPU_CUDA(cudaMemcpy(dst, &h, sizeof(h), cudaMemcpyHostToDevice));
  MGPU_CUDA(cudaMemset(dbar, 0, sizeof(unsigned long long)));
  MGPU_CUDA(cudaMemset(drec, 0, sizeof(MgpuIterRec)));
  KrylovArgs a{};
  a.n = n;
  a.row_ptr = drp;
  a.col = dcol;
  a.diag = ddiag;
  a.aval = dval;
  a.fval = dfval;
  a.b = db;
  a.x = dx;
  a.r = dkw;
  a.r0 = dkw + n;
  a.p = dkw + 2l * n;
  a.v = dkw + 3l * n;
  a.s = dkw + 4l * n;
  a.t = dkw + 5l * n;
  a.ph = dkw + 6l * n;
  a.sh = dkw + 7l * n;
  a.z = dkw + 8l * n;
  a.w = dkw + 9l * n;
  a.nlev_lo = L.nlo;
  a.lo_ptr = dlop;
  a.lo_rows = dlor;
  a.nlev_up = L.nup;
  a.up_ptr = dupp;
  a.up_rows = dupr;
  a.lt_pos = dmir;
  a.tol = tol;
  a.maxit = maxit;
  a.precond = precond;
  bool sweeps = false;
  if (precond != 1)
    TRY(plan_sweep(n, P.width, P.bw, L.nlo, dlop, dlor, L.nup, dupp, dupr, dferr, 0, sweeps));
  a.width = sweeps ? P.width : 0;
  a.bw = P.bw;
  a.zero_x = 0;
  a.mpi_mode = norm_mode ? 1 : 0;
  a.partials = dpart;
  a.bar = dbar;
  a.st = dst;
  a.recs = drec;
  a.slot = 0;
  a.ier_breakdown = 0;
  a.ferr = dferr;
  cudaStream_t s = 0;
  if (precond != 1) TRY(launch_factor(a, precond, s));
  if (bicg)
    TRY(launch_krylov_bicgstab(a, s));
  else
    TRY(launch_krylov_pcg(a, s));
  MGPU_CUDA(cudaDeviceSynchronize());
  MgpuIterRec r{};
  MGPU_CUDA(cudaMemcpy(&r, drec, sizeof(r), cudaMemcpyDeviceToHost));
  MGPU_CUDA(cudaMemcpy(&h, dst, sizeof(h), cudaMemcpyDeviceToHost));
  MGPU_CUDA(cudaMemcpy(x, dx, sizeof(double) * n, cudaMemcpyDeviceToHost));
  if (h.timeout) {
    set_error("a bounded device wait ran out (grid barrier)");
    return MGPU_E_TIMEOUT;
  }
  *it = r.lin_it[0];
  *res = r.lin_res[0];
  *ierr = r.lin_ierr[0];
  return 0;
}

int mgpu_pcg_poly_solve(int n, const int32_t* row_ptr, const int32_t* col_idx, const double* val, const double* b,
                        double* x, double tol, int maxit, int precision, int cheb_degree, int* it, double* res,
                        int* ierr) {
  if (n <= 0 || !row_ptr || !col_idx || !val || !b || !x || !it || !res || !ierr || maxit < 0 ||
      (precision != MGPU_PREC_MIXED && precision != MGPU_PREC_FP64_POLY) || n > kMixedMaxRows) {
    set_error("mgpu_pcg_poly_solve: invalid argument");
    return MGPU_E_ARG;
  }
  TRY(check_rows(n, row_ptr));
  DevBuf B;
  const size_t nz = row_ptr[n] - 1;
  TRY(B.reserve(32 * nz + 520 * (size_t)n + (1 << 18)));
  Pattern P;
  TRY(load_pattern(n, row_ptr, col_idx, B, P));
  *it = 0;
  *res = 0.0;
  *ierr = 0;
  if (!P.full_diag) {
    set_error("mgpu_pcg_poly_solve: a row has no diagonal entry");
    return MGPU_E_ARG;
  }
  int k = cheb_degree;
  double ratio = g_cheb_ratio;
  if (k <= 0) cheb_params(n, k, ratio);  // the tuning keys, as a case's pressure solve of n rows
  return precision == MGPU_PREC_MIXED ? poly_solve<float>(n, P, B, val, b, x, tol, maxit, k, ratio, it, res, ierr)
                                      : poly_solve<double>(n, P, B, val, b, x, tol, maxit, k, ratio, it, res, ierr);
}

int mgpu_csr_matvec(int n, const int32_t* row_ptr, const int32_t* col_idx, const double* val, const double* x,
                    double* y) {
  if (n <= 0 || !row_ptr || !col_idx || !val || !x || !y) {
    set_error("mgpu_csr_matvec: invalid argument");
    return MGPU_E_ARG;
  }
  std::vector<int> rp(n + 1);
  for (int i = 0; i <= n; ++i) rp[i] = row_ptr[i] - 1;
  const int nnz = rp[n];
  std::vector<int> col(nnz);
  for (int k = 0; k < nnz; ++k) col[k] = col_idx[k] - 1;
  DevBuf B;
  int *drp, *dcol;
  double *dval, *dx, *dy;
  TRY(B.up(drp, rp.data(), n + 1));
  TRY(B.up(dcol, col.data(), nnz));
  TRY(B.up(dval, val, nnz));
  TRY(B.up(dx, x, n));
  TRY(B.alloc(dy, n));
  TRY(launch_spmv(n, drp, dcol, dval, dx, dy, 0));
  MGPU_CUDA(cudaMemcpy(y, dy, sizeof(double) * n, cudaMemcpyDeviceToHost));
  return 0;
}

int mgpu_build_connectivity(const MgpuMesh* mesh, int32_t* cf_ptr, int32_t* cf, int32_t* c2c_ptr, int32_t* c2c,
                            int32_t* row_ptr, int32_t* col_idx, int32_t* nnz) {
  HostMesh m;
  std::string why;
  if (int e = load_host_mesh(mesh, m, why)) {
    set_error(why);
    return e;
  }
  HostTopo t;
  build_topology(m, t);
  for (int i = 0; i <= m.N; ++i) {
    cf_ptr[i] = t.cf_ptr[i] + 1;
    c2c_ptr[i] = t.c2c_ptr[i] + 1;
    row_ptr[i] = t.row_ptr[i] + 1;
  }
  for (size_t k = 0; k < t.cf.size(); ++k) cf[k] = t.cf[k] + 1;
  for (size_t k = 0; k < t.c2c.size(); ++k) c2c[k] = t.c2c[k] + 1;
  for (size_t k = 0; k < t.col.size(); ++k) col_idx[k] = t.col[k] + 1;
  *nnz = (int32_t)t.col.size();
  return 0;
}

int mgpu_geometry(const MgpuMesh* mesh, double* xf, double* sf, double* area, double* vol, double* xc,
                  double* lf) {
  HostMesh m;
  std::string why;
  if (int e = load_host_mesh(mesh, m, why)) {
    set_error(why);
    return e;
  }
  HostTopo t;
  build_topology(m, t);
  DevBuf B;
  DeviceCase d{};
  d.N = m.N;
  d.F = m.F;
  const long N = m.N, F = m.F;
  double *x, *pcen;
  int *fptr, *fnodes;
  TRY(B.up(d.c0, m.c0.data(), F));
  TRY(B.up(d.c1, m.c1.data(), F));
  TRY(B.up(d.cf_ptr, t.cf_ptr.data(), N + 1));
  TRY(B.up(d.cf, t.cf.data(), t.cf.size()));
  TRY(B.up(x, m.x.data(), m.x.size()));
  TRY(B.up(fptr, m.fptr.data(), m.fptr.size()));
  TRY(B.up(fnodes, m.fnodes.data(), m.fnodes.size()));
  TRY(B.alloc(pcen, 3 * N));
  TRY(B.alloc(d.xf, 3 * F));
  TRY(B.alloc(d.sf, 3 * F));
  TRY(B.alloc(d.area, F));
  TRY(B.alloc(d.lf, F));
  TRY(B.alloc(d.vol, N));
  TRY(B.alloc(d.xc, 3 * N));
  TRY(B.alloc(d.dn, F));
  TRY(B.alloc(d.dsf, F));
  TRY(B.alloc(d.Dm, F));
  TRY(B.alloc(d.tv, 3 * F));
  TRY(B.alloc(d.mnc, F));
  AsmParams P{};
  P.mu = 1.0;
  P.nonorth_corr = 1.0;
  TRY(geometry_setup(d, x, fptr, fnodes, pcen, P, 0));
  MGPU_CUDA(cudaDeviceSynchronize());
  auto down3 = [&](double* dst, const double* src, long n) -> int {
    std::vector<double> h(3 * n);
    MGPU_CUDA(cudaMemcpy(h.data(), src, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost));
    for (long i = 0; i < n; ++i)
      for (int k = 0; k < 3; ++k) dst[3 * i + k] = h[k * n + i];
    return 0;
  };
  TRY(down3(xf, d.xf, F));
  TRY(down3(sf, d.sf, F));
  TRY(down3(xc, d.xc, N));
  MGPU_CUDA(cudaMemcpy(area, d.area, sizeof(double) * F, cudaMemcpyDeviceToHost));
  MGPU_CUDA(cudaMemcpy(vol, d.vol, sizeof(double) * N, cudaMemcpyDeviceToHost));
  MGPU_CUDA(cudaMemcpy(lf, d.lf, sizeof(double) * F, cudaMemcpyDeviceToHost));
  return 0;
}

int mgpu_rcm_order(const MgpuMesh* mesh, int32_t* new_of_old) {
  HostMesh m;
  std::string why;
  if (!new_of_old) return MGPU_E_ARG;
  if (int e = load_host_mesh(mesh, m, why)) {
    set_error(why);
    return e;
  }
  std::vector<int> o;
  rcm_order(m, o);
  std::copy(o.begin(), o.end(), new_of_old);
  return 0;
}

}  // extern "C"
