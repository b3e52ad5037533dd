// Whole chains of small blocks in one launch.  Below ns ~ 64 a block's products are a
// few microseconds of FP64 work, less than the launches and the idle tails around
// them, so one cluster of CTAs walks the block columns and keeps what the next block
// needs in (distributed) shared memory.
#include <algorithm>

#include "rgf_device.h"
#include "rgf_internal.h"

namespace rgf {

namespace {

constexpr int CHAIN_THREADS = 256;

// How many neighbouring threads (a power of two up to MAX) share each of n elements of
// `terms` terms: the fewest FP64 instructions on an SM sub-partition.
template <int MAX>
__device__ __forceinline__ int lanes_per_element(int n, int terms) {
  int best = 1, cost = 1 << 30;
  for (int ks = 1, lg = 1; ks <= MAX; ks *= 2, ++lg) {
    const int c = ((n * ks + 31) / 32 + 3) / 4 * ((terms + ks - 1) / ks + lg);
    if (c < cost) {
      cost = c;
      best = ks;
    }
  }
  return best;
}

__host__ __device__ inline int odd(int x) { return x | 1; }

// Doubles of shared memory: S twice, K twice, and of the own columns Q twice and G.
__host__ __device__ inline size_t selinv_chain_elems(int ns, int m2, int nc) {
  const int own = (ns + nc - 1) / nc;
  return 2 * (size_t)m2 * odd(m2) + 2 * (size_t)ns * odd(m2) + 2 * (size_t)own * ns +
         (size_t)own * odd(m2);
}

// ---- selected inversion, blocks nt-1 .. 0 ----------------------------------------
// Per block, with S = [Sigma_{i+1,i+1}, .; Sigma_{d,i+1}, Sigma_dd] (symmetric, m2 = ns + nd;
// for the last block only its Sigma_dd part):
//   G = -S K (the rows below Sigma_ii), Sigma_ii = Q - K^T G, Q = U_i U_i^T.
// CTA q owns columns q, q + NC, ... of both products: G's are what its columns of
// Sigma_ii need, so the CTAs meet once a block, when the new S (both triangles) goes
// to every CTA's shared memory.  S is double-buffered: the buffer written for block i
// was last read for block i + 1, before the barrier in between.  K and the own
// columns of Q come by asynchronous copies one block ahead.  An element's terms are
// shared by up to eight threads so that all 256 work.
// One cluster's FP64 units bound it (1.5 ns m2^2 FMAs a block over NC SMs) from
// ns ~ 24, the exchange (~1.5 us a block) below.
// Selected inversion of 40 blocks, launches per block -> this: ns = 6 0.46 -> 0.13 ms,
// ns = 16 1.15 -> 0.15, ns = 32 0.84 -> 0.24, ns = 42 0.75 -> 0.41, ns = 64 0.97 -> 0.74
// (0.1 ms of each the inverses and K).
struct SelinvChain {
  int ns, nd;
  long long nt;
  const double* K;     // blocks 0 .. nt-2, m2 x ns each
  const double* Klast; // last block, nd x ns
  double* MS;          // Sigma in the factor's block positions; Q in its diagonal blocks
};

__global__ void __launch_bounds__(CHAIN_THREADS) selinv_chain_kernel(const SelinvChain p) {
  extern __shared__ double smem[];
  const int ns = p.ns, nd = p.nd, m2 = ns + nd, nc = gridDim.x, rank = blockIdx.x;
  const int tid = threadIdx.x;
  const int own = (ns + nc - 1) / nc;                     // most columns of a CTA
  const int ncol = ns > rank ? (ns - rank + nc - 1) / nc : 0;
  const int sp = odd(m2);                                 // pitch of S, K and G columns
  double* S0 = smem;
  double* K0 = S0 + 2 * m2 * sp;
  double* Q0 = K0 + 2 * ns * sp;
  double* G = Q0 + 2 * own * ns;                          // column j: rank + nc j
  const long long sP = (long long)ns * (2 * ns + nd);
  pdl_wait();
  auto fetch = [&](long long i) {  // K_i and the own columns of Q_i, lower part
    const bool last = i == p.nt - 1;
    const int r0 = last ? ns : 0, mm = m2 - r0;
    const double* src = last ? p.Klast : p.K + i * ns * m2;
    double* Kb = K0 + (i & 1) * ns * sp;
    for (int c = tid >> 5; c < ns; c += CHAIN_THREADS / 32)
      for (int r = tid & 31; r < mm; r += 32) cp_async8(Kb + c * sp + r0 + r, src + c * mm + r);
    const double* Q = p.MS + i * sP;
    const long long lda = last ? m2 : 2 * ns + nd;
    double* Qb = Q0 + (i & 1) * own * ns;
    for (int j = tid >> 5; j < ncol; j += CHAIN_THREADS / 32) {
      const int c = rank + nc * j;
      for (int r = c + (tid & 31); r < ns; r += 32) cp_async8(Qb + j * ns + r, Q + r + c * lda);
    }
    cp_async_commit();
  };
  fetch(p.nt - 1);
  {  // Sigma_dd into the first S
    const double* Sdd = p.MS + (p.nt - 1) * sP + (long long)ns * m2;
    double* S = S0 + ((p.nt - 1) & 1) * m2 * sp;
    for (int e = tid; e < 2 * nd * nd; e += CHAIN_THREADS) {
      const int x = e % (nd * nd);
      (e < nd * nd ? S : S0 + (p.nt & 1) * m2 * sp)[(ns + x / nd) * sp + ns + x % nd] = Sdd[x];
    }
  }
  __syncwarp();
  cluster_sync();  // every CTA is here before the first remote store
  for (long long i = p.nt - 1; i >= 0; --i) {
    const bool last = i == p.nt - 1;
    const int r0 = last ? ns : 0, mm = m2 - r0;
    double* D = p.MS + i * sP;
    const long long lda = last ? m2 : 2 * ns + nd;
    const double* S = S0 + (i & 1) * m2 * sp;             // of block i + 1
    double* Sn = S0 + ((i + 1) & 1) * m2 * sp;            // of this block
    const double* Kb = K0 + (i & 1) * ns * sp;
    const double* Qb = Q0 + (i & 1) * own * ns;
    cp_async_wait<0>();
    __syncthreads();
    if (i > 0) fetch(i - 1);
    {  // G, own columns
      const int n = ncol * mm, ks = lanes_per_element<8>(n, mm), t = tid & (ks - 1);
      for (int e0 = 0; e0 < n; e0 += CHAIN_THREADS / ks) {
        const int e = e0 + tid / ks;
        const bool live = e < n;
        if (!__any_sync(0xffffffffu, live)) continue;
        const int j = live ? e / mm : 0, r = live ? r0 + e - j * mm : r0;
        const double* k = Kb + (rank + nc * j) * sp;
        double a = 0.0;
        for (int l = r0 + t; l < m2; l += ks) a = fma(S[l * sp + r], k[l], a);
        for (int o = 1; o < ks; o *= 2) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (!live) continue;
        a = -a;
        if (t == 0) {
          G[j * sp + r] = a;
          D[ns + (r - r0) + (rank + nc * j) * lda] = a;
        }
        if (r >= ns && i > 0) {
          const int c = rank + nc * j;
          for (int z = t; z < nc; z += ks) {
            st_cluster(cluster_addr(Sn + c * sp + r, z), a);
            st_cluster(cluster_addr(Sn + r * sp + c, z), a);
          }
        }
      }
    }
    __syncthreads();
    {  // Sigma_ii, own columns, lower part
      int n = 0;
      for (int j = 0; j < ncol; ++j) n += ns - rank - nc * j;
      const int ks = lanes_per_element<8>(n, mm), t = tid & (ks - 1);
      for (int e0 = 0; e0 < n; e0 += CHAIN_THREADS / ks) {
        int e = e0 + tid / ks, j = 0, c = rank;
        const bool live = e < n;
        if (!__any_sync(0xffffffffu, live)) continue;
        if (!live) e = 0;
        while (e >= ns - c) {
          e -= ns - c;
          c += nc;
          ++j;
        }
        const int r = c + e;
        const double* k = Kb + r * sp;
        const double* g = G + j * sp;
        double a = 0.0;
        for (int l = r0 + t; l < m2; l += ks) a = fma(k[l], g[l], a);
        for (int o = 1; o < ks; o *= 2) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (!live) continue;
        a = Qb[j * ns + r] - a;
        if (t == 0) D[r + c * lda] = a;
        if (t == ks - 1 && r > c) D[c + r * lda] = a;
        if (i > 0)
          for (int z = t; z < nc; z += ks) {
            st_cluster(cluster_addr(Sn + c * sp + r, z), a);
            st_cluster(cluster_addr(Sn + r * sp + c, z), a);
          }
      }
    }
    __syncwarp();
    cluster_sync();
  }
  pdl_trigger();
}

// ---- block substitution: all right-hand sides through all blocks ---------------------
// Forward, then backward (U_i = L_ii^{-T}, F_i = L_{i+1,i}):
//   r_i = b_i - F_{i-1} y_{i-1},  y_i = U_i^T r_i;
//   x_d = U_d U_d^T (b_d - sum_i C_i y_i), the blocks of the sum dealt over the CTAs;
//   v_i = y_i - [F_i; C_i]^T [x_{i+1}; x_d],  x_i = U_i v_i.
// CTA q of the cluster owns h neighbouring rows of every block's vectors and computes
// them; each new vector goes to every CTA's shared memory, with one cluster
// barrier per product.  Its rows or columns of the matrices do not depend on the chain:
// they come by asynchronous copies one product ahead.
// A product is bound by its barrier and the latency of its reduction (~1.5-2 us), from
// ~8 K FMAs a CTA by the FP64 units.  Solves of 40 blocks, launches per product ->
// this, with one / eight right-hand sides: ns = 3 377 / 819 -> 153 / 167 us, ns = 64
// 446 / 1000 -> 279 / 398, ns = 128 556 / 1100 -> 347 / 785.
struct SolveChain {
  int ns, nd, nrhs;
  long long nt, n;
  const double *MF, *U;
  double *R, *Y;  // b, then x; y
};

// Rows of a CTA, and doubles of shared memory: two matrix slices, and the vectors.
__host__ __device__ inline int solve_rows(int ns, int nc) { return (ns + nc - 1) / nc; }
__host__ __device__ inline size_t solve_slice(int ns, int nd, int nc) {
  const int h = solve_rows(ns, nc);
  const size_t rows = (size_t)ns * odd(h), cols = (size_t)h * odd(ns + nd);
  return rows > cols ? rows : cols;
}
__host__ __device__ inline size_t solve_chain_elems(int ns, int nd, int nrhs, int nc) {
  return 2 * solve_slice(ns, nd, nc) + (size_t)nrhs * (2 * ns + nd + (nc + 2) * nd) +
         (size_t)nd * nd;
}

__global__ void __launch_bounds__(CHAIN_THREADS) solve_chain_kernel(const SolveChain p) {
  extern __shared__ double smem[];
  const int ns = p.ns, nd = p.nd, m2 = ns + nd, nq = p.nrhs, nc = gridDim.x, rank = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31;
  const int h = solve_rows(ns, nc), hp = odd(h), cp = odd(m2);
  const int lo = min(rank * h, ns), hi = min(lo + h, ns);  // own rows
  const size_t slice = solve_slice(ns, nd, nc);
  double* W = smem + 2 * slice;   // r_i, then v_i: ns a right-hand side
  double* Z = W + nq * ns;        // y_i, then [x_i; x_d]: m2
  double* T = Z + nq * m2;        // arrowhead: the CTAs' parts of the sum, nq x nd each
  double* T1 = T + nc * nq * nd;  // b_d - sum, then U_d^T of it
  double* T2 = T1 + nq * nd;
  double* Ud = T2 + nq * nd;
  const long long ss = (long long)ns * ns, sP = (long long)ns * (2 * ns + nd);
  int buf = 0;                    // slice buffer of the next product
  auto lda_of = [&](long long i) { return (long long)(i == p.nt - 1 ? ns : 2 * ns) + nd; };
  // rows [r0, r1) of a matrix with `terms` columns from c0: term l of row r at [l hp + r - r0]
  auto fetch_rows = [&](const double* A, long long ld, int r0, int r1, int c0, int terms) {
    double* d = smem + buf * slice;
    const int w = r1 - r0, g = w <= 16 ? 16 : 32;  // lanes along the rows
    for (int l = c0 + tid / g; l < terms; l += CHAIN_THREADS / g)
      for (int r = tid % g; r < w; r += g) cp_async8(d + l * hp + r, A + r0 + r + l * ld);
    cp_async_commit();
  };
  // columns [r0, r1) of a matrix, rows [0, len(r)): term l of column r at [(r - r0) cp + l]
  auto fetch_cols = [&](const double* A, long long ld, int r0, int r1, int terms, bool tri) {
    double* d = smem + buf * slice;
    for (int r = r0 + (tid >> 5); r < r1; r += CHAIN_THREADS / 32)
      for (int l = lane; l < (tri ? r + 1 : terms); l += 32)
        cp_async8(d + (r - r0) * cp + l, A + l + r * ld);
    cp_async_commit();
  };
  auto next = [&] {  // the slice of this product has arrived; the other buffer is free
    cp_async_wait<0>();
    __syncthreads();
    buf ^= 1;
    return smem + (buf ^ 1) * slice;
  };
  // out(r, q, init(r, q), sum over l in [l0(r), l1(r)) of a[(r - r0) rs + l ls] v[q vs + l],
  // t, ks) for rows [r0, r1) and every right-hand side; t is the thread's place among the
  // ks that share the element
  auto product = [&](const double* a, int rs, int ls, int r0, int r1, const double* v, int vs,
                     auto l0, auto l1, int terms, auto init, auto out) {
    const int n = (r1 - r0) * nq;
    const int ks = lanes_per_element<32>(n, terms);
    const int t = tid & (ks - 1);
    for (int e0 = 0; e0 < n; e0 += CHAIN_THREADS / ks) {
      const int e = e0 + tid / ks;
      const bool live = e < n;
      if (!__any_sync(0xffffffffu, live)) continue;
      const int q = live ? e / (r1 - r0) : 0, r = live ? r0 + e - q * (r1 - r0) : r0;
      const double* ar = a + (r - r0) * rs;
      const double* vq = v + q * vs;
      const double x0 = init(r, q);
      double s0 = 0.0, s1 = 0.0;
      int l = l0(r) + t;
      const int end = l1(r);
      for (; l + ks < end; l += 2 * ks) {
        s0 = fma(ar[l * ls], vq[l], s0);
        s1 = fma(ar[(l + ks) * ls], vq[l + ks], s1);
      }
      if (l < end) s0 = fma(ar[l * ls], vq[l], s0);
      s0 += s1;
      for (int o = 1; o < ks; o *= 2) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      if (live) out(r, q, x0, s0, t, ks);
    }
    __syncwarp();
  };
  auto to_all = [&](double* d, double x, int t, int ks) {
    for (int z = t; z < nc; z += ks) st_cluster(cluster_addr(d, z), x);
  };
  const auto zero = [](int) { return 0; };
  const auto all_m2 = [&](int) { return m2; };
  const auto all_ns = [&](int) { return ns; };
  const auto none = [](int, int) { return 0.0; };

  pdl_wait();
  fetch_cols(p.U, ns, lo, hi, ns, true);
  for (int e = tid; e < nq * ns; e += CHAIN_THREADS) W[e] = p.R[e % ns + (long long)(e / ns) * p.n];
  for (int e = tid; e < nq * nd; e += CHAIN_THREADS)
    T1[e] = p.R[p.nt * ns + e % nd + (long long)(e / nd) * p.n];
  for (int e = tid; e < nd * nd; e += CHAIN_THREADS) Ud[e] = p.U[p.nt * ss + e];
  __syncwarp();
  cluster_sync();  // every CTA is here before the first remote store

  // ---- forward ----
  for (long long i = 0; i < p.nt; ++i) {
    const bool last = i == p.nt - 1;
    // y_i = U_i^T r_i
    const double* a = next();
    if (!last) fetch_rows(p.MF + i * sP + ns, lda_of(i), lo, hi, 0, ns);
    product(a, cp, 1, lo, hi, W, ns, zero, [](int r) { return r + 1; }, ns, none,
            [&](int r, int q, double, double s, int t, int ks) {
              if (!last) to_all(Z + q * m2 + r, s, t, ks);
              if (t == 0) p.Y[i * ns + r + q * p.n] = s;
            });
    cluster_sync();
    if (last) break;
    // r_{i+1} = b_{i+1} - F_i y_i
    a = next();
    fetch_cols(p.U + (i + 1) * ss, ns, lo, hi, ns, true);
    product(a, 1, hp, lo, hi, Z, m2, zero, all_ns, ns,
            [&](int r, int q) { return p.R[(i + 1) * ns + r + q * p.n]; },
            [&](int r, int q, double b, double s, int t, int ks) {
              to_all(W + q * ns + r, b - s, t, ks);
            });
    cluster_sync();
  }
  // ---- the arrowhead ----
  fetch_cols(p.MF + (p.nt - 1) * sP + ns, ns + nd, lo, hi, nd, false);
  if (nd > 0) {
    for (int e = tid >> 5; e < nq * nd; e += CHAIN_THREADS / 32) {
      const int q = e / nd, d = e % nd;
      double s = 0.0;
      for (long long i = rank; i < p.nt; i += nc) {
        const long long ld = lda_of(i);
        const double* C = p.MF + i * sP + ld - nd + d;
        const double* y = p.Y + i * ns + q * p.n;
#pragma unroll 4
        for (int l = lane; l < ns; l += 32) s = fma(C[l * ld], y[l], s);
      }
      for (int o = 1; o < 32; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
      for (int z = lane; z < nc; z += 32) st_cluster(cluster_addr(T + rank * nq * nd + e, z), s);
    }
    __syncwarp();
    cluster_sync();
    for (int e = tid; e < nq * nd; e += CHAIN_THREADS) {
      double s = 0.0;
      for (int z = 0; z < nc; ++z) s += T[z * nq * nd + e];
      T1[e] -= s;
    }
    __syncthreads();
    for (int e = tid; e < nq * nd; e += CHAIN_THREADS) {  // x_d = U_d (U_d^T t), in every CTA
      const int q = e / nd, r = e % nd;
      double s = 0.0;
      for (int l = 0; l <= r; ++l) s = fma(Ud[r * nd + l], T1[q * nd + l], s);
      T2[e] = s;
    }
    __syncthreads();
    for (int e = tid; e < nq * nd; e += CHAIN_THREADS) {
      const int q = e / nd, r = e % nd;
      double s = 0.0;
      for (int l = nd - 1; l >= r; --l) s = fma(Ud[l * nd + r], T2[q * nd + l], s);
      Z[q * m2 + ns + r] = s;
      if (rank == 0) p.R[p.nt * ns + r + q * p.n] = s;
    }
  }
  // ---- backward ----
  for (long long i = p.nt - 1; i >= 0; --i) {
    const bool last = i == p.nt - 1;
    // v_i = y_i - [F_i; C_i]^T [x_{i+1}; x_d]
    const double* a = next();
    fetch_rows(p.U + i * ss, ns, lo, hi, lo, ns);
    const int s0 = last ? ns : 0;
    product(a - s0, cp, 1, lo, hi, Z, m2, [&](int) { return s0; }, all_m2, m2 - s0,
            [&](int r, int q) { return p.Y[i * ns + r + q * p.n]; },
            [&](int r, int q, double y, double s, int t, int ks) {
              to_all(W + q * ns + r, y - s, t, ks);
            });
    cluster_sync();
    // x_i = U_i v_i
    a = next();
    if (i > 0) fetch_cols(p.MF + (i - 1) * sP + ns, lda_of(i - 1), lo, hi, m2, false);
    product(a, 1, hp, lo, hi, W, ns, [](int r) { return r; }, all_ns, ns, none,
            [&](int r, int q, double, double s, int t, int ks) {
              if (i > 0) to_all(Z + q * m2 + r, s, t, ks);
              if (t == 0) p.R[i * ns + r + q * p.n] = s;
            });
    if (i > 0) cluster_sync();
  }
  pdl_trigger();
  __syncwarp();
  cluster_sync();  // no CTA leaves while another may still store to it
}

}  // namespace

// One CTA does blocks of up to 12 rows as fast as eight (the FP64 work of a block is
// below the exchange), eight up to 28, then sixteen.  The line at 72 (56 with clusters
// of eight): a block at ns = 42 / 56 / 64 / 72 takes 8.5 / 11 / 17 / 22 us in the chain
// with 16 CTAs, 17 / 21 / 23 / 24 in launches of its own.
int selinv_chain_ctas(const BtaShape& sh) {
  const long long m2 = sh.ns + sh.nd;
  if (m2 > SELINV_CHAIN_MAX) return 0;
  static const int widest = widest_cluster(
      selinv_chain_kernel, sizeof(double) * selinv_chain_elems(SELINV_CHAIN_MAX, SELINV_CHAIN_MAX, 8),
      CHAIN_THREADS);
  if (!widest || (widest < 16 && m2 > 56)) return 0;
  return m2 <= 12 ? 1 : m2 <= 28 ? 8 : widest;
}

void launch_selinv_chain(const BtaShape& sh, int nc, const double* K, const double* Klast,
                         double* MS, cudaStream_t s) {
  const int ns = (int)sh.ns, m2 = (int)(sh.ns + sh.nd);
  const size_t bytes = selinv_chain_elems(ns, m2, nc) * sizeof(double);
  allow_wide_clusters(selinv_chain_kernel, SELINV_CHAIN_SMEM);  // an attribute of the current device
  launch_k_cluster(selinv_chain_kernel, dim3(nc), dim3(CHAIN_THREADS), dim3(nc), bytes, s,
                   SelinvChain{ns, (int)sh.nd, sh.nt, K, Klast, MS});
}

// The lines, from solves of 40 to 60 blocks (chain of 16 CTAs / separate products, in
// us): ns = 128 347 / 490 with one right-hand side, 781 / 960 with eight; ns = 160 458 / 456
// with one, 606 / 565 with two; ns = 256 875 / 812.  One CTA beats eight while a
// product has up to ~600 FMAs (ns = 3: 153 against 195), sixteen beat eight from ~48 rows.
// Past 16 right-hand sides the separate products spread over the whole GPU, and the chain
// is the better way only up to ~8 K FMAs and 256 results of a CTA a product (chain /
// products in ms: ns = 3, nt = 60 0.85 / 0.99 with 256, 1.43 / 1.1 with 512; ns = 16, nt = 60
// 0.86 / 1.06 with 128, 1.25 / 1.10 with 192; ns = 64, nt = 40 0.68 / 0.74 with 24, 1.24 / 0.90
// with 64; ns = 144, nt = 30 1.16 / 0.82 with 17, 3.3 / 1.3 with 64).
int solve_chain_ctas(const BtaShape& sh, int nrhs) {
  const long long m2 = sh.ns + sh.nd;
  if (m2 > SOLVE_CHAIN_MAX || sh.ns > (nrhs == 1 ? 176 : 144)) return 0;
  static const int widest = widest_cluster(solve_chain_kernel, SOLVE_CHAIN_SMEM, CHAIN_THREADS);
  if (!widest || (widest < 16 && sh.ns > 100)) return 0;
  const int nc = m2 * m2 * nrhs <= 600 ? 1 : m2 <= 48 ? 8 : widest;
  if (nrhs > 16 &&
      (sh.ns * sh.ns * nrhs > 8192LL * nc || solve_rows((int)sh.ns, nc) * (long long)nrhs > 256))
    return 0;
  if (solve_chain_elems((int)sh.ns, (int)sh.nd, nrhs, nc) * sizeof(double) > SOLVE_CHAIN_SMEM) return 0;
  return nc;
}

void launch_solve_chain(const BtaShape& sh, int nc, const double* MF, const double* U, double* R,
                        double* Y, int nrhs, cudaStream_t s) {
  allow_wide_clusters(solve_chain_kernel, SOLVE_CHAIN_SMEM);  // an attribute of the current device
  launch_k_cluster(solve_chain_kernel, dim3(nc), dim3(CHAIN_THREADS), dim3(nc),
                   solve_chain_elems((int)sh.ns, (int)sh.nd, nrhs, nc) * sizeof(double), s,
                   SolveChain{(int)sh.ns, (int)sh.nd, nrhs, sh.nt, sh.n, MF, U, R, Y});
}

}  // namespace rgf
