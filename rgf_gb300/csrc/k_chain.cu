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

__device__ __forceinline__ void cp_async8(void* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
               :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// How many neighbouring threads (1, 2, 4 or 8) share each of n elements of `terms` terms:
// the fewest FP64 instructions of a thread, over all rounds of the CTA's threads.
__device__ __forceinline__ int lanes_per_element(int n, int terms) {
  int best = 1, cost = 1 << 30;
  for (int ks = 1, lg = 0; ks <= 8; ks *= 2, ++lg) {
    const int c = (n * ks + CHAIN_THREADS - 1) / CHAIN_THREADS * ((terms + ks - 1) / ks + lg + 1);
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
      const int n = ncol * mm, ks = lanes_per_element(n, mm), t = tid & (ks - 1);
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
      const int ks = lanes_per_element(n, mm), t = tid & (ks - 1);
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

}  // namespace rgf
