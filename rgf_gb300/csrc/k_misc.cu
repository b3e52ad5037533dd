// Memory-bound kernels of the RGF recursion: CSC ingest into the block
// layout, reductions, diagonal extraction, residual SpMV and small helpers.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "rgf_device.h"
#include "rgf_internal.h"

namespace rgf {

// Block-column layout (the reference's MF, RGF.H:95, 114-138):
// block column i < nt-1 is (2ns+nd) x ns = [L_ii; L_{i+1,i}; C_i],
// block column nt-1 is (ns+nd) x ns = [L_ii; C_i], the corner is nd x nd.
__host__ __device__ inline long long col_offset_d(long long ns, long long nt, long long nd,
                                                  long long i) {
  if (i < nt) return i * ns * (2 * ns + nd);
  return (nt - 1) * ns * (2 * ns + nd) + ns * (ns + nd);
}
__host__ __device__ inline long long lda_d(long long ns, long long nt, long long nd, long long i) {
  if (i < nt - 1) return 2 * ns + nd;
  if (i < nt) return ns + nd;
  return nd;
}
__host__ __device__ inline long long dense_row_d(long long ns, long long nt, long long i) {
  if (i < nt - 1) return 2 * ns;
  if (i == nt - 1) return ns;
  return 0;
}

long long mf_col_offset(const BtaShape& sh, long long i) { return col_offset_d(sh.ns, sh.nt, sh.nd, i); }
long long mf_lda(const BtaShape& sh, long long i) { return lda_d(sh.ns, sh.nt, sh.nd, i); }
long long mf_dense_row(const BtaShape& sh, long long i) { return dense_row_d(sh.ns, sh.nt, i); }

namespace {

// One warp per CSC column: the column's block column and panel offset are
// computed once, then every entry maps to a row of that panel.  Follows the
// mapping of the reference's getPos (CWC_utility.cu:998-1029) without its
// per-entry linear column search (CWC_utility.cu:1093-1095).
__global__ void ingest_kernel(BtaShape sh, long long c_lo, long long c_hi,
                              const size_t* __restrict__ ia, const size_t* __restrict__ ja,
                              const double* __restrict__ a, double* __restrict__ MF,
                              DevStatus* st) {
  pdl_wait();
  pdl_trigger();
  const long long c = c_lo + (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= c_hi) return;
  const long long ns = sh.ns, nt = sh.nt, nd = sh.nd, n = sh.n;
  const long long ib = c < ns * nt ? c / ns : nt;
  const long long jc = ib < nt ? c - ib * ns : c - nt * ns;
  const long long off = col_offset_d(ns, nt, nd, ib);
  const long long lda = lda_d(ns, nt, nd, ib);
  const long long ro = dense_row_d(ns, nt, ib);
  const size_t e0 = ia[c], e1 = ia[c + 1];
  bool bad = false;
  for (size_t e = e0 + lane; e < e1; e += 32) {
    const long long r = (long long)ja[e];
    bool ok = r >= c && r < n;
    long long row = 0;
    if (ok) {
      const long long rb = r < ns * nt ? r / ns : nt;
      if (rb == ib) row = (ib < nt) ? r - ib * ns : r - nt * ns;
      else if (rb == ib + 1 && rb < nt) row = r - ib * ns;
      else if (rb == nt) row = ro + (r - nt * ns);
      else ok = false;
    }
    if (ok) MF[off + jc * lda + row] = a[e];
    else bad = true;
  }
  if (bad) atomicOr(&st->bad_input, 1);
}

// log of every diagonal entry of the factor MF; each block of 256 columns sums
// its logs in a fixed tree order into parts[block]
__global__ void diag_log_kernel(BtaShape sh, const double* MF, double* parts) {
  pdl_wait();
  pdl_trigger();
  __shared__ double v[256];
  const long long k = (long long)blockIdx.x * 256 + threadIdx.x;
  double x = 0.0;
  if (k < sh.n) {
    const long long ns = sh.ns, nt = sh.nt, nd = sh.nd;
    long long pos;
    if (k < ns * nt) {
      const long long i = k / ns, j = k - i * ns;
      pos = col_offset_d(ns, nt, nd, i) + j * (lda_d(ns, nt, nd, i) + 1);
    } else {
      const long long j = k - ns * nt;
      pos = col_offset_d(ns, nt, nd, nt) + j * (nd + 1);
    }
    x = log(MF[pos]);
  }
  v[threadIdx.x] = x;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) v[threadIdx.x] += v[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) parts[blockIdx.x] = v[0];
}

__global__ void logdet_reduce_kernel(const double* parts, int nparts, double* out) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x;
  double s = 0.0;
  for (int i = lane; i < nparts; i += 32) s += parts[i];
  __shared__ double ws[32];
  ws[lane] = s;
  __syncwarp();
  if (lane == 0) {
    double t = 0.0;
    for (int i = 0; i < 32; ++i) t += ws[i];
    *out = 2.0 * t;
  }
}

__global__ void extract_diag_kernel(BtaShape sh, const double* MS, double* diag) {
  pdl_wait();
  pdl_trigger();
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= sh.n) return;
  const long long ns = sh.ns, nt = sh.nt, nd = sh.nd;
  long long pos;
  if (k < ns * nt) {
    const long long i = k / ns, j = k - i * ns;
    pos = col_offset_d(ns, nt, nd, i) + j * (lda_d(ns, nt, nd, i) + 1);
  } else {
    const long long j = k - ns * nt;
    pos = col_offset_d(ns, nt, nd, nt) + j * (nd + 1);
  }
  diag[k] = MS[pos];
}

__global__ void set_identity_kernel(double* X, long long ld, int m, long long stride) {
  pdl_wait();
  pdl_trigger();
  X += (long long)blockIdx.z * stride;
  const int r = blockIdx.x * 32 + threadIdx.x, c = blockIdx.y * 8 + threadIdx.y;
  if (r < m && c < m) X[r + (long long)c * ld] = (r == c) ? 1.0 : 0.0;
}

// X(r, c) = X(c, r) for r < c: the strictly upper triangle of the n x n matrix X
// (column-major, ld) from its lower one, and with S the full symmetric
// [X, Xd^T; Xd, Sdd] into S (packed; nd = 0: X alone).  Tiles of 32: nb of the rows
// of X, then those of the nd arrowhead rows.  The CTA of source tile (bi, bj),
// bi >= bj, reads it along its columns into shared memory and writes it transposed
// along the columns of tile (bj, bi); no CTA reads a tile another one writes.
__global__ void mirror_sigma_kernel(double* X, long long ld, int n, const double* Xd,
                                    const double* Sdd, int nd, double* S, int nb) {
  __shared__ double t[32][33];  // t[column offset][row offset] of the source tile
  pdl_wait();
  pdl_trigger();
  const int bi = blockIdx.x, bj = blockIdx.y;
  if (bi < bj) return;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  const bool dr = bi >= nb, dc = bj >= nb;       // arrowhead rows, columns
  const int r0 = (dr ? bi - nb : bi) * 32, c0 = (dc ? bj - nb : bj) * 32;
  const int nr = dr ? nd : n, nc = dc ? nd : n;
  const double* src = dc ? Sdd : dr ? Xd : X;
  const long long lds = dc ? nd : ld;
  const long long m2 = n + nd;
  const int fr = dr ? n : 0, fc = dc ? n : 0;  // where the tile's rows, columns start in S
  for (int k = ty; k < 32; k += 8) {
    const int r = r0 + tx, c = c0 + k;
    if (r < nr && c < nc && (dr != dc || r >= c)) {
      const double v = src[r + (long long)c * lds];
      t[k][tx] = v;
      if (S) S[fr + r + (fc + c) * m2] = v;
    }
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    const int r = c0 + tx, c = r0 + k;  // the transposed element (r, c) = t[tx][k]
    if (r >= nc || c >= nr || (dr == dc && r >= c)) continue;
    if (!dr) X[r + (long long)c * ld] = t[tx][k];
    if (S) S[fc + r + (fr + c) * m2] = t[tx][k];
  }
}

// y = A x with A symmetric, stored as its lower CSC: column c contributes
// a_rc x_c to y_r (scatter) and, off the diagonal, a_rc x_r to y_c (gather).
// Entries outside the lower triangle (r < c) or past the last row (r >= n)
// are skipped, so every write stays inside y[0, n); when `bad` is given such
// an entry also sets *bad.
__global__ void sym_spmv_kernel(long long n, const size_t* __restrict__ ia,
                                const size_t* __restrict__ ja, const double* __restrict__ a,
                                const double* __restrict__ x, double* y, int* bad) {
  pdl_wait();
  pdl_trigger();
  const long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= n) return;
  const double xc = x[c];
  double g = 0.0;
  bool skipped = false;
  for (size_t e = ia[c] + lane; e < ia[c + 1]; e += 32) {
    const size_t ru = ja[e];
    if (ru < (size_t)c || ru >= (size_t)n) {
      skipped = true;
      continue;
    }
    const long long r = (long long)ru;
    const double v = a[e];
    atomicAdd(&y[r], v * xc);
    if (r != c) g += v * x[r];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
  if (lane == 0 && g != 0.0) atomicAdd(&y[c], g);
  if (skipped && bad) atomicExch(bad, 1);
}

// Y[:, q] = A X[:, q] for q < nrhs (<= N <= SPMV_MAX_RHS, columns n apart): the
// product of sym_spmv_kernel for several right-hand sides in one pass over
// the CSC (each entry is read once for all of them).  The CSC must be valid
// (the handle's, which ingest checked).
// Bound by the FP64 units (a multiplication and an FMA an entry and right-hand side; a
// predicated-off one costs the same, so the count is a template parameter): eight right-hand sides, 8 M entries 411 -> 304 us.
template <int N>
__global__ void sym_spmv_multi_kernel(long long n, const size_t* __restrict__ ia,
                                      const size_t* __restrict__ ja,
                                      const double* __restrict__ a,
                                      const double* __restrict__ X, double* Y, int nrhs) {
  pdl_wait();
  pdl_trigger();
  const long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= n) return;
  double xc[N], g[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    xc[q] = q < nrhs ? X[q * n + c] : 0.0;
    g[q] = 0.0;
  }
  for (size_t e = ia[c] + lane; e < ia[c + 1]; e += 32) {
    const long long r = (long long)ja[e];
    const double v = a[e];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      if (q < nrhs) {
        atomicAdd(&Y[q * n + r], v * xc[q]);
        if (r != c) g[q] += v * X[q * n + r];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < N; ++q) {
    double t = g[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0 && q < nrhs && t != 0.0) atomicAdd(&Y[q * n + c], t);
  }
}

// out[0] = ||b - y||_2, out[1] = ||b||_2 of right-hand side blockIdx.y (columns n apart,
// results 2 apart; a cluster along x).  As in dnrm2, the sums of squares are scaled so
// that neither overflows nor underflows: a first pass finds max |b - y| and max |b|
// (order-independent), a second sums the squares of the entries scaled by the power of
// two just above each maximum (exact scaling), in a fixed tree order and then in rank
// order.  If *bad is set (an index was out of range in the product) both are NaN.
// One launch for all right-hand sides, each over up to 8 CTAs; one CTA and one launch
// each took 8 x 0.15 ms at n = 50 004.
__device__ __forceinline__ double pow2_below_inv(double mx) {
  // 2^-e with 2^(e-1) <= mx < 2^e (mx > 0 and finite), so mx * 2^-e is in [0.5, 1)
  int e = 0;
  frexp(mx, &e);
  return ldexp(1.0, -e);
}

constexpr int NORM_THREADS = 512;
__global__ void __launch_bounds__(NORM_THREADS)
    residual_norm_kernel(long long n, const double* b, const double* y, double* out, const int* bad,
                         const double* rres = nullptr) {
  __shared__ double s1[NORM_THREADS], s2[NORM_THREADS];
  __shared__ double part[2][2];  // [pass][residual, b] of this CTA
  pdl_wait();
  pdl_trigger();
  const int t = threadIdx.x, nc = gridDim.x, rank = blockIdx.x;
  b += blockIdx.y * n;
  if (y) y += blockIdx.y * n;
  if (rres) rres += blockIdx.y * n;
  out += 2 * blockIdx.y;
  double m1 = 0.0, m2 = 0.0;
  // r_i = b_i - y_i, or rres[i] when the residual is given
  auto res = [&](long long i) { return rres ? rres[i] : b[i] - y[i]; };
  const long long i0 = (long long)rank * NORM_THREADS + t, di = (long long)nc * NORM_THREADS;
  for (long long i = i0; i < n; i += di) {
    m1 = fmax(m1, fabs(res(i)));
    m2 = fmax(m2, fabs(b[i]));
  }
  auto reduce = [&](double v1, double v2, double* of, auto op) {
    s1[t] = v1;
    s2[t] = v2;
    __syncthreads();
    for (int w = NORM_THREADS / 2; w > 0; w >>= 1) {
      if (t < w) {
        s1[t] = op(s1[t], s1[t + w]);
        s2[t] = op(s2[t], s2[t + w]);
      }
      __syncthreads();
    }
    if (t == 0) {
      of[0] = s1[0];
      of[1] = s2[0];
    }
    __syncthreads();
    cluster_sync();
    double a1 = ld_cluster(of, 0), a2 = ld_cluster(of + 1, 0);
    for (int z = 1; z < nc; ++z) {
      a1 = op(a1, ld_cluster(of, z));
      a2 = op(a2, ld_cluster(of + 1, z));
    }
    m1 = a1;
    m2 = a2;
  };
  reduce(m1, m2, part[0], [](double u, double v) { return fmax(u, v); });
  const double mr = m1, mb = m2;
  const bool fr = mr > 0.0 && isfinite(mr), fb = mb > 0.0 && isfinite(mb);
  const double sr = fr ? pow2_below_inv(mr) : 1.0, sb = fb ? pow2_below_inv(mb) : 1.0;
  double r2 = 0.0, b2 = 0.0;
  for (long long i = i0; i < n; i += di) {
    const double r = res(i) * sr, bb = b[i] * sb;
    r2 += r * r;
    b2 += bb * bb;
  }
  reduce(r2, b2, part[1], [](double u, double v) { return u + v; });
  if (rank == 0 && t == 0) {
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    const bool invalid = bad && *bad;
    out[0] = invalid ? nan : (fr ? sqrt(m1) / sr : mr);
    out[1] = invalid ? nan : (fb ? sqrt(m2) / sb : mb);
  }
  cluster_sync();  // a CTA's parts are read until every CTA is here
}

// partial[q][p] = sum_j C_i(a, j) C_i(b, j) for the pairs p = (a >= b), over the cells (block
// column i, 256 of its columns) q, q + gridDim.x, ...; one warp per pair, fixed-order warp
// reduction.  One launch at the end of the factorization instead of a product per block
// column beside it (nt launches of ~10 us on the look-ahead stream).  At most
// ARROW_SYRK_CTAS partial sums of a pair, eight CTAs an SM: their memory (5 MB at 32 rows)
// does not grow with nt past that.
constexpr int ARROW_CHUNK = 256, ARROW_SYRK_CTAS = 8 * GB300_SMS;
__global__ void __launch_bounds__(256)
    arrow_syrk_kernel(BtaShape sh, const double* MF, double* partial) {
  pdl_wait();
  pdl_trigger();
  const long long ns = sh.ns, nt = sh.nt, nd = sh.nd;
  const long long per = (ns + ARROW_CHUNK - 1) / ARROW_CHUNK, cells = nt * per;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pairs = (int)(nd * (nd + 1) / 2);
  double* out = partial + (long long)blockIdx.x * pairs;
  for (int p = warp; p < pairs; p += 8) {
    int a = 0, b = p;
    while (b > a) b -= ++a;  // p = a (a + 1) / 2 + b
    double s = 0.0;
    for (long long cell = blockIdx.x; cell < cells; cell += gridDim.x) {
      const long long i = cell / per, j0 = (cell - i * per) * ARROW_CHUNK;
      const long long j1 = min(ns, j0 + ARROW_CHUNK), lda = lda_d(ns, nt, nd, i);
      const double* Cb = MF + col_offset_d(ns, nt, nd, i) + dense_row_d(ns, nt, i);
      for (long long j = j0 + lane; j < j1; j += 32) s = fma(Cb[a + j * lda], Cb[b + j * lda], s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[p] = s;
  }
}

// corner(a, b) -= the partial sums, one warp per pair
__global__ void arrow_syrk_reduce_kernel(BtaShape sh, const double* partial, long long chunks,
                                         double* MF) {
  pdl_wait();
  pdl_trigger();
  const long long nd = sh.nd;
  const int pairs = (int)(nd * (nd + 1) / 2);
  const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (p >= pairs) return;
  double s = 0.0;
  for (long long c = lane; c < chunks; c += 32) s += partial[c * pairs + p];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  int a = 0, b = p;
  while (b > a) b -= ++a;
  if (lane == 0) MF[col_offset_d(sh.ns, sh.nt, nd, sh.nt) + a + b * nd] -= s;
}

// partial[i][q][dd] = sum_j C_i(dd, j) * rhs_i(j, q): one CTA per block
// column i, one warp per (dd, q) pair, fixed-order warp reduction.
__global__ void arrow_gemv_kernel(BtaShape sh, const double* MF, const double* rhs, long long ldr,
                                  int nrhs, double* partial) {
  pdl_wait();
  pdl_trigger();
  const long long i = blockIdx.x;
  const long long ns = sh.ns, nt = sh.nt, nd = sh.nd;
  const double* Cb = MF + col_offset_d(ns, nt, nd, i) + dense_row_d(ns, nt, i);
  const long long lda = lda_d(ns, nt, nd, i);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int p = blockIdx.y * nw + warp; p < nd * nrhs; p += gridDim.y * nw) {
    const int dd = p % nd, q = p / nd;
    const double* R = rhs + i * ns + (long long)q * ldr;
    double s = 0.0;
    for (long long j = lane; j < ns; j += 32) s += Cb[dd + j * lda] * R[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) partial[(i * nrhs + q) * nd + dd] = s;
  }
}

__global__ void arrow_reduce_kernel(BtaShape sh, const double* partial, int nrhs, double* rhs,
                                    long long ldr) {
  pdl_wait();
  pdl_trigger();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const long long nd = sh.nd;
  if (p >= nd * nrhs) return;
  const int dd = p % nd, q = p / nd;
  double s = 0.0;
  for (long long i = 0; i < sh.nt; ++i) s += partial[(i * nrhs + q) * nd + dd];
  rhs[sh.nt * sh.ns + dd + (long long)q * ldr] -= s;
}

}  // namespace

void launch_ingest(const BtaShape& sh, const size_t* ia, const size_t* ja, const double* a,
                   double* MF, DevStatus* st, cudaStream_t s, long long c_lo, long long c_hi) {
  if (c_hi < 0) c_hi = sh.n;
  if (c_hi <= c_lo) return;
  const long long threads = (c_hi - c_lo) * 32;
  const int bs = 256;
  launch_k(ingest_kernel, dim3((unsigned)((threads + bs - 1) / bs)), dim3(bs), 0, s, sh, c_lo,
           c_hi, ia, ja, a, MF, st);
}

int logdet_parts(const BtaShape& sh) { return (int)((sh.n + 255) / 256); }

void launch_logdet(const BtaShape& sh, const double* MF, double* parts, double* out,
                   cudaStream_t s) {
  const int np = logdet_parts(sh);
  launch_k(diag_log_kernel, dim3(np), dim3(256), 0, s, sh, MF, parts);
  launch_k(logdet_reduce_kernel, dim3(1), dim3(32), 0, s, parts, np, out);
}

long long selinv_chunk(const BtaShape& sh) {
  const long long one = (long long)sizeof(double) * (sh.ns + sh.nd) * sh.ns;
  return std::max(1LL, std::min(sh.nt - 1, (long long)K_CHUNK_BYTES / one));
}

void launch_extract_diag(const BtaShape& sh, const double* MS, double* diag, cudaStream_t s) {
  launch_k(extract_diag_kernel, dim3((unsigned)((sh.n + 255) / 256)), dim3(256), 0, s, sh, MS,
           diag);
}

void launch_set_identity(double* X, long long ld, int m, int batch, long long stride,
                         cudaStream_t s) {
  if (m <= 0 || batch <= 0) return;
  dim3 grid((m + 31) / 32, (m + 7) / 8, batch);
  launch_k(set_identity_kernel, grid, dim3(32, 8), 0, s, X, ld, m, stride);
}

void launch_mirror_sigma(double* X, long long ld, int n, const double* Xd, const double* Sdd,
                         int nd, double* S, cudaStream_t s) {
  if (!S) {
    nd = 0;
    if (n <= 1) return;
  }
  const unsigned nb = (unsigned)((n + 31) / 32), all = nb + (unsigned)((nd + 31) / 32);
  launch_k(mirror_sigma_kernel, dim3(all, all), dim3(32, 8), 0, s, X, ld, n, Xd, Sdd, nd, S, (int)nb);
}

// r = b - y; x += d (element-wise over len entries)
__global__ void sub_kernel(long long len, const double* b, const double* y, double* r) {
  pdl_wait();
  pdl_trigger();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < len) r[i] = b[i] - y[i];
}
__global__ void add_kernel(long long len, double* x, const double* d) {
  pdl_wait();
  pdl_trigger();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < len) x[i] += d[i];
}

void launch_residual_vectors(long long n, int nrhs, const size_t* ia, const size_t* ja,
                             const double* a, const double* X, const double* B, double* Y,
                             double* R, cudaStream_t s) {
  cudaMemsetAsync(Y, 0, sizeof(double) * n * nrhs, s);
  const long long threads = n * 32;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  for (int q0 = 0; q0 < nrhs; q0 += SPMV_MAX_RHS) {  // the CSC is read once per 16 RHS
    const int k = std::min(SPMV_MAX_RHS, nrhs - q0);
    auto* kern = k <= 1   ? sym_spmv_multi_kernel<1>
                 : k <= 2 ? sym_spmv_multi_kernel<2>
                 : k <= 3 ? sym_spmv_multi_kernel<3>
                 : k <= 4 ? sym_spmv_multi_kernel<4>
                 : k <= 6 ? sym_spmv_multi_kernel<6>
                 : k <= 8 ? sym_spmv_multi_kernel<8>
                 : k <= 12 ? sym_spmv_multi_kernel<12>
                          : sym_spmv_multi_kernel<16>;
    launch_k(kern, dim3(grid), dim3(256), 0, s, n, ia, ja, a, X + q0 * n, Y + q0 * n, k);
  }
  const long long len = n * nrhs;
  launch_k(sub_kernel, dim3((unsigned)((len + 255) / 256)), dim3(256), 0, s, len, B, Y, R);
}

// CTAs that share one right-hand side's norms: 4096 entries each
static void launch_norms(long long n, int nrhs, const double* B, const double* Y, double* out,
                         const int* bad, const double* R, cudaStream_t s) {
  unsigned nc = 1;
  while (nc < 8 && n > nc * 4096LL) nc *= 2;
  launch_k_cluster(residual_norm_kernel, dim3(nc, nrhs), dim3(NORM_THREADS), dim3(nc), 0, s, n, B, Y,
                   out, bad, R);
}

void launch_rhs_norms(long long n, int nrhs, const double* R, const double* B, double* out,
                      cudaStream_t s) {
  if (nrhs > 0) launch_norms(n, nrhs, B, nullptr, out, nullptr, R, s);
}

void launch_add(long long len, double* x, const double* d, cudaStream_t s) {
  launch_k(add_kernel, dim3((unsigned)((len + 255) / 256)), dim3(256), 0, s, len, x, d);
}

cudaError_t launch_residual(long long n, const size_t* ia, const size_t* ja, const double* a,
                            const double* x, const double* b, double* scratch, double* out,
                            int* bad, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(double) * n, s);
  if (e == cudaSuccess && bad) e = cudaMemsetAsync(bad, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  const long long threads = n * 32;
  launch_k(sym_spmv_kernel, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, s, n, ia, ja,
           a, x, scratch, bad);
  launch_norms(n, 1, b, scratch, out, bad, nullptr, s);
  return cudaGetLastError();
}

static long long arrow_partials(const BtaShape& sh) {
  return std::min<long long>(sh.nt * ((sh.ns + ARROW_CHUNK - 1) / ARROW_CHUNK), ARROW_SYRK_CTAS);
}
long long arrow_syrk_elems(const BtaShape& sh) {
  return arrow_partials(sh) * (sh.nd * (sh.nd + 1) / 2);
}
void launch_arrow_syrk(const BtaShape& sh, double* MF, double* partial, cudaStream_t s) {
  const long long parts = arrow_partials(sh);
  const int pairs = (int)(sh.nd * (sh.nd + 1) / 2);
  launch_k(arrow_syrk_kernel, dim3((unsigned)parts), dim3(256), 0, s, sh, (const double*)MF, partial);
  launch_k(arrow_syrk_reduce_kernel, dim3((pairs + 7) / 8), dim3(256), 0, s, sh,
           (const double*)partial, parts, MF);
}

void launch_arrow_gemv(const BtaShape& sh, const double* MF, const double* rhs, long long ldr,
                       int nrhs, double* partial, cudaStream_t s) {
  if (sh.nd <= 0) return;
  const unsigned pairs = (unsigned)std::min<long long>((sh.nd * nrhs + 7) / 8, 32);  // a warp each
  launch_k(arrow_gemv_kernel, dim3((unsigned)sh.nt, pairs), dim3(256), 0, s, sh, MF, rhs, ldr, nrhs,
           partial);
}

void launch_arrow_reduce(const BtaShape& sh, const double* partial, int nrhs, double* rhs,
                         long long ldr, cudaStream_t s) {
  if (sh.nd <= 0) return;
  const int p = (int)(sh.nd * nrhs);
  launch_k(arrow_reduce_kernel, dim3((p + 127) / 128), dim3(128), 0, s, sh, partial, nrhs, rhs, ldr);
}

}  // namespace rgf
