// FP64 kernels of the RGF recursion for sm_103a.
//
// On GB300 the FP64 rate is the same for DMMA (mma.sync .f64) and DFMA
// (about 1 TFLOP/s per GPU), so the FP64 GEMM below is bound by the FP64
// pipe, not by memory: 64x64 output tiles, 4 warps of 32x32 built from
// m8n8k4 DMMA fragments, operands staged through shared memory with a
// register prefetch of the next K slice.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>

#include "rgf_device.h"
#include "rgf_internal.h"

namespace rgf {

namespace {

__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

struct GemmTileRange {
  int klo, khi;
};

template <int TM, int TK>
__device__ __forceinline__ GemmTileRange k_range(const GemmDesc& g, int m0, int n0) {
  int klo = 0, khi = g.k;
  if (g.triA == TRI_LOWER) khi = min(khi, m0 + TM);
  if (g.triA == TRI_UPPER) klo = max(klo, m0);
  if (g.triB == TRI_LOWER) klo = max(klo, n0);
  if (g.triB == TRI_UPPER) khi = min(khi, n0 + TM);
  klo = (klo / TK) * TK;
  return {klo, khi};
}

// TM x TM output tiles, 4 warps of (TM/2) x (TM/2) built from m8n8k4 DMMA
// fragments, K staged TK at a time.  TM = 64, TK = 16 for large products;
// TM = 32, TK = 8 spreads small products over four times as many CTAs (each
// SM retires only ~3.5 FP64 flops per cycle, so a small product on few SMs
// is slow however short it is).
template <int TM, int TK>
__global__ void __launch_bounds__(128, TM == 64 ? 3 : 8) gemm_fp64_kernel(GemmDesc g) {
  constexpr int F = TM / 16;             // 8 x 8 fragments per warp side
  constexpr int LPT = TM * TK / 128;     // elements per thread per operand and stage
  constexpr int PAD = TM + 4;
  pdl_wait();
  // blockIdx.x counts the written tiles only, column by column.  (With a CTA for every
  // tile the skipped ones' places were dealt out too, and SMs got two of the others while
  // some got none: the lower half of 333 x 333 x 338 in 132 CTAs 110 us, now 65.)
  const TilePos tile = tile_at(g.outLower, (g.m + TM - 1) / TM, blockIdx.x);
  const int m0 = tile.x * TM, n0 = tile.y * TM;
  // blockIdx.z = batch item * ksplit + K slice; the slices of a tile are a cluster
  const bool splitk = g.ksplit > 1;
  const long long bz = blockIdx.z / g.ksplit;
  const int kz = (int)blockIdx.z - (int)bz * g.ksplit;
  const double* __restrict__ A = g.A + bz * g.sA;
  const double* A2 = g.A2 ? g.A2 + bz * g.sA - g.mA1 : nullptr;
  const int mA1 = g.A2 ? g.mA1 : g.m;
  const double* __restrict__ B = g.B + bz * g.sB;
  const double* C = g.C ? g.C + bz * g.sC : nullptr;
  double* D = g.D + bz * g.sD;
  const double* C2 = g.C2 ? g.C2 + bz * g.sC - g.mD1 : nullptr;
  double* D2 = g.D2 ? g.D2 + bz * g.sD - g.mD1 : nullptr;
  const int mD1 = g.D2 ? g.mD1 : g.m;

  // operand tiles, then (split K) this slice's sums, element (r, c) at [c * TM + r]
  constexpr int SMEM = 2 * TK * PAD > TM * TM ? 2 * TK * PAD : TM * TM;
  __shared__ double smem[SMEM];
  double(*As)[PAD] = reinterpret_cast<double(*)[PAD]>(smem);
  double(*Bs)[PAD] = reinterpret_cast<double(*)[PAD]>(smem + TK * PAD);

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int wm = (warp & 1) * (TM / 2), wn = (warp >> 1) * (TM / 2);
  GemmTileRange kr = k_range<TM, TK>(g, m0, n0);
  if (splitk) {
    const int len = max(0, kr.khi - kr.klo);
    const int chunk = ((len + g.ksplit - 1) / g.ksplit + TK - 1) / TK * TK;
    const int lo = kr.klo + kz * chunk;
    kr.khi = min(kr.khi, lo + chunk);
    kr.klo = lo;
  }

  double acc[F][F][2];
#pragma unroll
  for (int i = 0; i < F; ++i)
#pragma unroll
    for (int j = 0; j < F; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  double ra[LPT], rb[LPT];
  auto load = [&](int kt) {
#pragma unroll
    for (int j = 0; j < LPT; ++j) {
      int rr, kk;
      if (!g.transA) { rr = tid % TM; kk = tid / TM + (128 / TM) * j; }
      else           { kk = tid % TK; rr = tid / TK + (128 / TK) * j; }
      const int r = m0 + rr, kg = kt + kk;
      bool ok = r < g.m && kg < kr.khi;
      if (g.triA == TRI_LOWER) ok = ok && kg <= r;
      if (g.triA == TRI_UPPER) ok = ok && kg >= r;
      double v = 0.0;
      if (ok) v = g.transA ? A[(long long)kg + (long long)r * g.lda]
                           : (r < mA1 ? A : A2)[(long long)r + (long long)kg * g.lda];
      ra[j] = v;
    }
#pragma unroll
    for (int j = 0; j < LPT; ++j) {
      int cc, kk;
      if (!g.transB) { kk = tid % TK; cc = tid / TK + (128 / TK) * j; }
      else           { cc = tid % TM; kk = tid / TM + (128 / TM) * j; }
      const int c = n0 + cc, kg = kt + kk;
      bool ok = c < g.n && kg < kr.khi;
      if (g.triB == TRI_LOWER) ok = ok && kg >= c;
      if (g.triB == TRI_UPPER) ok = ok && kg <= c;
      double v = 0.0;
      if (ok) v = g.transB ? B[(long long)c + (long long)kg * g.ldb] : B[(long long)kg + (long long)c * g.ldb];
      rb[j] = v;
    }
  };
  auto store = [&]() {
#pragma unroll
    for (int j = 0; j < LPT; ++j) {
      if (!g.transA) As[tid / TM + (128 / TM) * j][tid % TM] = ra[j];
      else           As[tid % TK][tid / TK + (128 / TK) * j] = ra[j];
      if (!g.transB) Bs[tid % TK][tid / TK + (128 / TK) * j] = rb[j];
      else           Bs[tid / TM + (128 / TM) * j][tid % TM] = rb[j];
    }
  };

  // U U^T of upper triangular U runs its K range downwards: the leading terms (on U's
  // diagonal) come last, so that one addition rounds at the size of the result instead
  // of one per K step (relative error of Sigma at ns = 333: 7.5e-16 -> 5.9e-16)
  const bool down = g.triA == TRI_UPPER && g.triB == TRI_LOWER;
  if (kr.klo < kr.khi) {
    const int tiles = (kr.khi - kr.klo + TK - 1) / TK, kflip = down ? TK - 4 : 0;
    int kt = down ? kr.klo + (tiles - 1) * TK : kr.klo;
    load(kt);
    for (int it = 0; it < tiles; ++it) {
      store();
      __syncthreads();
      const int kn = down ? kt - TK : kt + TK;
      if (it + 1 < tiles) load(kn);
#pragma unroll
      for (int k4 = 0; k4 < TK; k4 += 4) {
        const int ks = k4 ^ kflip;
        if (kt + ks >= kr.khi) continue;  // a short last K tile: no products of the zero padding
        double af[F], bf[F];
#pragma unroll
        for (int i = 0; i < F; ++i) af[i] = As[ks + (lane & 3)][wm + i * 8 + (lane >> 2)];
#pragma unroll
        for (int j = 0; j < F; ++j) bf[j] = Bs[ks + (lane & 3)][wn + j * 8 + (lane >> 2)];
#pragma unroll
        for (int i = 0; i < F; ++i)
#pragma unroll
          for (int j = 0; j < F; ++j) dmma_8x8x4(acc[i][j], af[i], bf[j]);
      }
      kt = kn;
      __syncthreads();
    }
  }
  pdl_trigger();

  if (splitk) {
    // the slices' sums meet through distributed shared memory, in slice order;
    // each CTA writes its share of the tile
#pragma unroll
    for (int i = 0; i < F; ++i)
#pragma unroll
      for (int j = 0; j < F; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          smem[(wn + j * 8 + (lane & 3) * 2 + e) * TM + wm + i * 8 + (lane >> 2)] = acc[i][j][e];
    const int share = (TM * TM / 128 + g.ksplit - 1) / g.ksplit;  // passes of 128 elements
    constexpr int U = 4;                                          // passes in flight
    // only the passes there are issue FP64 instructions, alpha = +-1 takes none, and C is
    // on its way before the exchange (selected inversion at ns = 128, nt = 40 1.75 -> 1.69
    // ms, ns = 333, nt = 17 4.69 -> 4.64)
    bool met = false;
#pragma unroll 1
    for (int q0 = 0; q0 < share; q0 += U) {
      const int nu = min(U, share - q0);
      double v[U] = {}, cv[U];
      double* out[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = (kz * share + q0 + u) * 128 + tid;
        const int r = m0 + idx % TM, c = n0 + idx / TM;
        const bool ok = u < nu && idx < TM * TM && r < g.m && c < g.n && !(g.outLower && r < c);
        out[u] = ok ? (r < mD1 ? D : D2) + (long long)r + (long long)c * g.ldd : nullptr;
        cv[u] = 0.0;
        if (ok && g.beta != 0.0) cv[u] = (r < mD1 ? C : C2)[(long long)r + (long long)c * g.ldc];
      }
      if (!met) cluster_sync();
      met = true;
#pragma unroll 4
      for (int z = 0; z < g.ksplit; ++z) {
        double w[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          w[u] = ld_cluster(smem + min((kz * share + q0 + u) * 128 + tid, TM * TM - 1), z);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (u >= nu) break;
          v[u] += w[u];
          __syncwarp();
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (u >= nu) break;
        double x = v[u];
        if (g.alpha == -1.0) {
          x = -x;
        } else if (g.alpha != 1.0) {
          x *= g.alpha;
          __syncwarp();
        }
        if (g.beta != 0.0) {
          x = fma(g.beta, cv[u], x);
          __syncwarp();
        }
        if (out[u]) *out[u] = x;
      }
    }
    __syncwarp();
    cluster_sync();  // a CTA's sums are read until every CTA is here
    return;
  }
#pragma unroll
  for (int i = 0; i < F; ++i) {
    const int r = m0 + wm + i * 8 + (lane >> 2);
    if (r >= g.m) continue;
    const double* Cr = r < mD1 ? C : C2;
    double* Dr = r < mD1 ? D : D2;
#pragma unroll
    for (int j = 0; j < F; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = n0 + wn + j * 8 + (lane & 3) * 2 + e;
        if (c >= g.n) continue;
        if (g.outLower && r < c) continue;
        double v = g.alpha * acc[i][j][e];
        if (g.beta != 0.0) v += g.beta * Cr[(long long)r + (long long)c * g.ldc];
        Dr[(long long)r + (long long)c * g.ldd] = v;
      }
    }
  }
}

// Row-parallel triangular solve with a <= 64 x 64 lower tile:
// MODE 0: X := X L^{-T}, x_j = (b_j - sum_{l<j} x_l L_jl) / L_jj
// MODE 1: X := X L^{-1}, x_j = (b_j - sum_{l>j} x_l L_lj) / L_jj
// G lanes share one row; lane q of them keeps the unknowns t G + q in registers.
// The tile is held with its rows (MODE 1: columns) scaled to a unit diagonal, so
// step j hands z_j = x_j L_jj on with one shuffle and updates the unknowns after it
// with one FMA per slot; the slots are unrolled by blocks of G steps, so that no
// FP64 instruction is issued for a slot that is done (predicated off it costs
// the same).  G = 32 (4 rows a CTA) while that many CTAs fit the SMs a few times
// over, 8 (16 rows a CTA, fewer instructions a row) for more rows: the 64 rows of
// an inverse's leaf took 36 us with G = 8 and predicated slots, now ~19.
// INV: X = L^{-T} (b = I, MODE 0) of every 64-column diagonal tile of an nbk x nbk
// factor at once (blockIdx.z: the tile; X and L start at the first one).
template <int MODE, int G, bool INV = false>
__global__ void __launch_bounds__(128) trsm_rows_kernel(double* X, long long xrs, long long xcs,
                                                         int rows, const double* L, long long ldl,
                                                         int nbk, long long sX, long long sL) {
  constexpr int T = 64 / G;  // slots
  __shared__ double Ls[64][65];  // [j][l]: multiplier of z_j in unknown l
  __shared__ double rinv[64];
  pdl_wait();
  X += (long long)blockIdx.y * sX;
  L += (long long)blockIdx.y * sL;
  if (INV) {
    const int off = blockIdx.z * 64;
    X += off * (xcs + xrs);
    L += off * (ldl + 1);
    nbk = rows = min(64, nbk - off);
  }
  const int tid = threadIdx.x;
  if (tid < 64) rinv[tid] = tid < nbk ? 1.0 / L[(long long)tid * (ldl + 1)] : 0.0;
  const int lane = tid & 31, q = lane & (G - 1), gbase = lane & ~(G - 1);
  const long long r = (long long)blockIdx.x * (128 / G) + tid / G;
  const bool live = r < rows;
  double u[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int l = t * G + q;
    if (INV) u[t] = r == l ? 1.0 : 0.0;
    else u[t] = live && l < nbk ? X[r * xrs + (long long)l * xcs] : 0.0;
  }
  __syncthreads();
  for (int idx = tid; idx < nbk * 64; idx += 128) {
    const int c = idx >> 6, row = idx & 63;  // L(row, c), row >= c
    double v = 0.0;
    if (row > c && row < nbk) v = L[row + (long long)c * ldl];
    if (MODE == 0) Ls[c][row] = v * rinv[c];  // z_c -> unknown row
    else Ls[row][c] = v * rinv[row];          // z_row -> unknown c
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < T; ++b) {
    const int t0 = MODE == 0 ? b : T - 1 - b;  // slot being solved
#pragma unroll 1
    for (int s = 0; s < G; ++s) {
      const int jj = MODE == 0 ? s : G - 1 - s, j = t0 * G + jj;
      if (j >= nbk) {
        if (MODE == 0) break;
        continue;
      }
      const double z = -__shfl_sync(0xffffffffu, u[t0], gbase | jj);
      const double nv = fma(z, Ls[j][t0 * G + q], u[t0]);
      u[t0] = (MODE == 0 ? q > jj : q < jj) ? nv : u[t0];
#pragma unroll
      for (int t = MODE == 0 ? t0 + 1 : 0; t < (MODE == 0 ? T : t0); ++t)
        u[t] = fma(z, Ls[j][t * G + q], u[t]);
    }
  }
  pdl_trigger();
#pragma unroll
  for (int t = 0; t < T; ++t) {
    const int l = t * G + q;
    const double x = u[t] * rinv[l];
    if (live && l < nbk) X[r * xrs + (long long)l * xcs] = x;
  }
}

// Thin products (m <= 16, op(B) = B^T; the arrowhead rows): lane = output
// column, M (a template parameter: an absent row's FMA would cost as much as
// a present one's) accumulators per lane.  K is split over a cluster and the
// four warps as in gemm_thin_n_kernel below; B is read along its contiguous
// columns, A's M terms per k are one uniform load each.
template <int M>
__global__ void __launch_bounds__(128) gemm_thin_m_kernel(GemmDesc g, int kchunk) {
  __shared__ double part[4][M][32];
  __shared__ double red[M * 32];
  pdl_wait();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 32, c = c0 + lane;
  int k0 = blockIdx.y * kchunk, k1 = min(g.k, k0 + kchunk);
  if (g.triB == TRI_LOWER) k0 = max(k0, c0);        // op(B)(k, c) = 0 for k < c
  if (g.triB == TRI_UPPER) k1 = min(k1, c0 + 32);   // and for k > c
  const long long ras = g.transA ? g.lda : 1, kas = g.transA ? 1 : g.lda;
  double acc[M];
#pragma unroll
  for (int r = 0; r < M; ++r) acc[r] = 0.0;
  constexpr int U = 8;  // K terms in flight per warp
  for (int kt = k0 + w * U; kt < k1; kt += 4 * U) {
    double b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = kt + u;
      bool ok = k < k1 && c < g.n;
      if (g.triB == TRI_LOWER) ok = ok && k >= c;
      if (g.triB == TRI_UPPER) ok = ok && k <= c;
      b[u] = ok ? g.B[c + (long long)k * g.ldb] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (kt + u >= k1) break;
      const double* a = g.A + (kt + u) * kas;
#pragma unroll
      for (int r = 0; r < M; ++r) acc[r] = fma(r < g.m ? a[r * ras] : 0.0, b[u], acc[r]);
    }
  }
  pdl_trigger();
#pragma unroll
  for (int r = 0; r < M; ++r) part[w][r][lane] = acc[r];
  __syncthreads();
  for (int o = threadIdx.x; o < M * 32; o += 128) {
    const int r = o >> 5, l = o & 31;
    red[o] = ((part[0][r][l] + part[1][r][l]) + part[2][r][l]) + part[3][r][l];
  }
  const int nk = gridDim.y, rank = blockIdx.y;
  if (nk > 1) cluster_sync();
  else __syncthreads();
  for (int o = rank * 128 + threadIdx.x; o < M * 32; o += nk * 128) {
    const int r = o >> 5, col = c0 + (o & 31);
    double v = 0.0;
    if (nk > 1) {
      double part[8];  // all loads in flight, then the sum in rank order
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < nk) part[q] = ld_cluster(red + o, q);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q >= nk) break;
        v += part[q];
      }
    } else {
      v = red[o];
    }
    if (r < g.m && col < g.n) {
      v *= g.alpha;
      const bool hi = g.D2 && r >= g.mD1;
      const long long ro = hi ? r - g.mD1 : r;
      if (g.beta != 0.0) v += g.beta * (hi ? g.C2 : g.C)[ro + (long long)col * g.ldc];
      (hi ? g.D2 : g.D)[ro + (long long)col * g.ldd] = v;
    }
  }
  if (nk > 1) cluster_sync();
}

// Thin products (n <= 16, op(B) = B; the steps of the block substitution):
// bound by the FP64 units (m k n FMAs at ~0.55 TFMA/s; an FP64 instruction
// holds its unit ~76 cycles even with every lane predicated off, so the
// columns are a template parameter and no FMA is issued for absent ones).
// A CTA owns 32 output rows, lane = row.  A cluster of up to 8 CTAs
// (blockIdx.y) splits the rows' K range evenly, and the four warps a CTA's share (K
// tiles of 32 dealt to the warps left three of four FP64 units idle at K = 256): many SMs
// work on even a small product.  The partial sums
// meet in shared memory, first over the warps, then over the cluster through
// distributed shared memory, both in a fixed order: one launch per product.
// op(A) is read along its contiguous dimension; a transposed A goes through a
// per-warp 32 x 32 shared-memory tile.  Measured over whole solves (four such
// products per block column), against 128-row tiles with 16 predicated columns
// and a second launch for the reduction: one right-hand side at ns = 256,
// nt = 60 10.15 -> 0.81 ms (42 -> 3.4 us a product), eight 3.66 -> 2.01 ms by the even
// shares alone; eight at ns = 1000, nt = 50, split (with the residuals) 20.7 -> 7.8 ms.
// op(A) may be triangular: K tiles that lie in its other triangle are skipped.
// With `early` (the caller vouches that the previous kernel of the stream does not write
// A: the block substitution, whose matrices are the factor's) the first tile of A is
// loaded while that kernel still runs (eight right-hand sides, ns = 256, nt = 60:
// 2.01 -> 1.65 ms; one 0.90 -> 0.81).
// More columns than N go as groups of N (blockIdx.z; launch_gemm_thin_groups).
constexpr int THIN_KT = 32;  // K terms of one warp's tile
template <int N>
__global__ void __launch_bounds__(128) gemm_thin_n_kernel(GemmDesc g) {
  // per warp: tile of a transposed A, element (k, row) at [k][row ^ k] (no bank
  // conflicts either way, within the 48 KiB of N = 16); then the warps' sums
  __shared__ double At[4][THIN_KT][32];
  __shared__ double Bs[4][THIN_KT][N];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (N >= 8) {  // (smaller ones have no groups)
    const int first = blockIdx.z * N;  // column of this group of N
    g.n -= first;
    g.B += first * g.ldb;
    g.C += first * g.ldc;
    g.D += first * g.ldd;
  }
  // the row tiles with the longest K range go first
  const int bx = g.triA == TRI_LOWER ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const int r0 = bx * 32, r = r0 + lane;
  int k0 = 0, k1 = g.k;
  if (g.triA == TRI_LOWER) k1 = min(k1, r0 + 32);  // op(A)(r, kk) = 0 for kk > r
  if (g.triA == TRI_UPPER) k0 = min(k1, r0);       // and for kk < r
  // even shares of that range: of the cluster's CTAs (multiples of 8), of the warps (of 4)
  const int nk = gridDim.y, rank = blockIdx.y;  // the cluster spans blockIdx.y
  const int share = ((k1 - k0 + nk - 1) / nk + 7) & ~7;
  k0 = min(k1, k0 + rank * share);
  k1 = min(k1, k0 + share);
  const int part = ((k1 - k0 + 3) / 4 + 3) & ~3;
  k0 = min(k1, k0 + w * part);
  k1 = min(k1, k0 + part);
  double acc[N];
#pragma unroll
  for (int c = 0; c < N; ++c) acc[c] = 0.0;
  double ra[THIN_KT];  // op(A)(r, kt + kk), or (transposed) op(A)(r0 + kk, kt + lane)
  auto load_a = [&](int kt) {
    const int kn = min(THIN_KT, k1 - kt);
    if (!g.transA) {
      const double* a = g.A + r + (long long)kt * g.lda;
#pragma unroll
      for (int kk = 0; kk < THIN_KT; ++kk) {
        bool ok = kk < kn && r < g.m;
        if (g.triA == TRI_LOWER) ok = ok && kt + kk <= r;
        if (g.triA == TRI_UPPER) ok = ok && kt + kk >= r;
        ra[kk] = ok ? *a : 0.0;
        a += g.lda;
      }
    } else {
      const int kg = kt + lane;
      const double* a = g.A + kg + (long long)r0 * g.lda;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        bool ok = lane < kn && r0 + i < g.m;
        if (g.triA == TRI_LOWER) ok = ok && kg <= r0 + i;
        if (g.triA == TRI_UPPER) ok = ok && kg >= r0 + i;
        ra[i] = ok ? *a : 0.0;
        a += g.lda;
      }
    }
  };
  if (g.early && k0 < k1) load_a(k0);
  pdl_wait();
  if (!g.early && k0 < k1) load_a(k0);
  for (int kt = k0; kt < k1; kt += THIN_KT) {
    const int kn = min(THIN_KT, k1 - kt);
#pragma unroll
    for (int c = 0; c < N; ++c)
      Bs[w][lane][c] = lane < kn && c < g.n ? g.B[kt + lane + (long long)c * g.ldb] : 0.0;
    if (g.transA) {
#pragma unroll
      for (int i = 0; i < 32; ++i) At[w][lane][i ^ lane] = ra[i];
    }
    __syncwarp();
    if (g.transA) {
      for (int kk = 0; kk < kn; ++kk) {
        const double a = At[w][kk][lane ^ kk];
#pragma unroll
        for (int c = 0; c < N; ++c) acc[c] = fma(a, Bs[w][kk][c], acc[c]);
      }
    } else {
#pragma unroll
      for (int kk = 0; kk < THIN_KT; ++kk) {
        if (kk >= kn) break;
#pragma unroll
        for (int c = 0; c < N; ++c) acc[c] = fma(ra[kk], Bs[w][kk][c], acc[c]);
      }
    }
    __syncwarp();
    if (kt + THIN_KT < k1) load_a(kt + THIN_KT);
  }
  pdl_trigger();
  // this CTA's sums: warp partials in At[w][c][lane], summed in warp order
  // into red[c][row]
  __syncthreads();
#pragma unroll
  for (int c = 0; c < N; ++c) At[w][c][lane] = acc[c];
  __syncthreads();
  double* red = &Bs[0][0][0];  // N x 32
  for (int o = threadIdx.x; o < N * 32; o += 128) {
    const int c = o >> 5, l = o & 31;
    red[o] = ((At[0][c][l] + At[1][c][l]) + At[2][c][l]) + At[3][c][l];
  }
  if (nk > 1) cluster_sync();
  else __syncthreads();
  // the cluster's total in rank order; the outputs are dealt over its CTAs
  for (int o = rank * 128 + threadIdx.x; o < N * 32; o += nk * 128) {
    const int c = o >> 5, row = r0 + (o & 31);
    double v = 0.0;
    if (nk > 1) {
      double part[8];  // all loads in flight, then the sum in rank order
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < nk) part[q] = ld_cluster(red + o, q);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q >= nk) break;
        v += part[q];
      }
    } else {
      v = red[o];
    }
    if (row < g.m && c < g.n) {
      v *= g.alpha;
      if (g.beta != 0.0) v += g.beta * g.C[row + (long long)c * g.ldc];
      g.D[row + (long long)c * g.ldd] = v;
    }
  }
  if (nk > 1) cluster_sync();  // a CTA's sums are read until every CTA is here
}

// How many clusters of k CTAs the device holds with one CTA to an SM (asked of the
// runtime once, for a CTA that takes most of an SM's shared memory).
struct ClusterRoom {
  int clusters[9];
};
const ClusterRoom& cluster_room() {
  static const ClusterRoom room = [] {
    ClusterRoom r{};
    r.clusters[1] = GB300_SMS;
    auto* k = gemm_fp64_kernel<32, 8>;
    constexpr int FILL = 160 << 10;
    const bool ok =
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, FILL) == cudaSuccess;
    for (int n = 2; n <= 8; ++n) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(1, 1, n);
      cfg.blockDim = dim3(128);
      cfg.dynamicSmemBytes = FILL;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = n;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      if (!ok || cudaOccupancyMaxActiveClusters(&r.clusters[n], k, &cfg) != cudaSuccess)
        r.clusters[n] = 128 / n;
    }
    cudaGetLastError();
    return r;
  }();
  return room;
}

// K over 1, 2, 4 or 8 CTAs of a cluster: `least` K terms per CTA are the
// least worth a CTA of their own (a quarter of them per warp).
dim3 thin_split(const GemmDesc& g, int least, int* kchunk) {
  int kc = 1;
  while (kc < 8 && kc * least < g.k) kc *= 2;
  *kchunk = ((g.k + kc - 1) / kc + THIN_KT - 1) / THIN_KT * THIN_KT;
  return dim3(1, kc);
}
// (a thin-n CTA is worth 64 FMA instructions: 16 a warp, ~0.6 us)
template <int N>
void launch_thin_n(const GemmDesc& g, cudaStream_t s) {
  const int rows = (g.m + 31) / 32, groups = (g.n + N - 1) / N;
  int kc = 1;
  while (kc < 8 && g.k * N > kc * 64 && g.k > kc * 8) kc *= 2;
  while (groups > 1 && kc > 1 && rows * groups * kc > 4 * GB300_SMS) kc /= 2;
  launch_k_cluster(gemm_thin_n_kernel<N>, dim3(rows, kc, groups), dim3(128), dim3(1, kc), 0, s, g);
}
// Block substitution with THIN_N_MAX < n <= THIN_GROUPS_MAX right-hand sides: groups of 8 columns
// (12 from 193 on at up to 160 rows: 100, 40, 256 2.9 ms against 3.5 by eights; 200, 30, 256
// 4.8 against 3.9), K over a cluster only while that leaves four CTAs an SM.  Against 32-wide
// tiles, whose few K slices of 32 x 32 outputs fill little of the GPU, and 64-wide tiles
// with up to 16 slices through a workspace before them, whole solves (ns, nt and
// right-hand sides; this / 32-wide / before, in ms): 160, 30, 17 0.83 / 1.53 / 1.20;
// 256, 20, 64 1.6 / 2.2 / 1.7; 144, 30, 64 1.3 / 1.7 / 1.4; 512, 10, 32 1.1 / 1.6 / 1.3;
// 1000, 6, 128 5.5 / 5.8 / 6.8; 64, 40, 256 1.7 / 1.9 / 1.9.  Groups of 16 leave fewer CTAs
// (256, 20, 17: 1.1 against 0.81), and past 512 the tiles read A less often
// (nor do they pay below 8 rows).
constexpr int THIN_N_MAX = 16, THIN_GROUPS_MAX = 512;
void launch_gemm_thin_groups(const GemmDesc& g, cudaStream_t s) {
  if (g.n <= 192 || g.m > 160) launch_thin_n<8>(g, s);
  else launch_thin_n<12>(g, s);
}
template <int M>
void launch_thin_m(const GemmDesc& g, cudaStream_t s) {
  int kchunk;
  const dim3 cl = thin_split(g, THIN_KT, &kchunk);
  launch_k_cluster(gemm_thin_m_kernel<M>, dim3((g.n + 31) / 32, cl.y), dim3(128), cl, 0, s, g,
                   kchunk);
}
void launch_gemm_thin_n(const GemmDesc& g, cudaStream_t s) {
  if (g.n <= 1) launch_thin_n<1>(g, s);
  else if (g.n <= 2) launch_thin_n<2>(g, s);
  else if (g.n <= 3) launch_thin_n<3>(g, s);
  else if (g.n <= 4) launch_thin_n<4>(g, s);
  else if (g.n <= 6) launch_thin_n<6>(g, s);
  else if (g.n <= 8) launch_thin_n<8>(g, s);
  else if (g.n <= 12) launch_thin_n<12>(g, s);
  else launch_thin_n<16>(g, s);
}
void launch_gemm_thin_m(const GemmDesc& g, cudaStream_t s) {
  if (g.m <= 1) launch_thin_m<1>(g, s);
  else if (g.m <= 2) launch_thin_m<2>(g, s);
  else if (g.m <= 3) launch_thin_m<3>(g, s);
  else if (g.m <= 4) launch_thin_m<4>(g, s);
  else if (g.m <= 6) launch_thin_m<6>(g, s);
  else if (g.m <= 8) launch_thin_m<8>(g, s);
  else if (g.m <= 12) launch_thin_m<12>(g, s);
  else launch_thin_m<16>(g, s);
}

}  // namespace

double gemm_flops(const GemmDesc& g) {
  double m = g.m, n = g.n, k = g.k;
  double f = 2.0 * m * n * k;
  if (g.triA != TRI_NONE) f = m * (m + 1.0) * n;
  if (g.triB != TRI_NONE) f = m * n * (n + 1.0);
  if (g.outLower && g.m >= g.n && g.n > 0) f = 2.0 * k * (n * (n + 1.0) / 2.0 + (m - n) * n);
  return f * g.batch;
}

int launch_gemm_fp64(const GemmDesc& g0, cudaStream_t s) {
  if (g0.m <= 0 || g0.n <= 0 || g0.batch <= 0) return 0;
  GemmDesc g = g0;
  if (g.m <= 16 && g.transB && g.triA == TRI_NONE && g.batch == 1 && !g.outLower &&
      !g.A2) {
    launch_gemm_thin_m(g, s);
    return 1;
  }
  if (g.n <= (g.early && g.m >= 8 ? THIN_GROUPS_MAX : THIN_N_MAX) && !g.transB && g.triB == TRI_NONE &&
      g.batch == 1 && !g.outLower && !g.A2 && !g.D2) {
    if (g.n <= THIN_N_MAX) launch_gemm_thin_n(g, s);
    else launch_gemm_thin_groups(g, s);
    return 1;
  }
  // Output tile and split K (a cluster of up to 8 CTAs): the kernel is bound by
  // the FP64 units, so a launch lasts as long as the SM with the most work:
  // ceil(CTAs / 152) shares of tile^2 K / ksplit FMAs at 3200 a microsecond and
  // SM, at least two where the tiles' clusters do not fit the chip one CTA to an
  // SM; split K costs ~2 us.  32-wide tiles leave less of a last share empty than
  // 64-wide ones and were never slower (FP64 factorize + RGFdiag at ns = 1000,
  // nt = 10 81 against 115 ms, ns = 333, nt = 17 12.2 against 16.8).  Against the
  // previous rule (up to 16 K slices of 64-wide tiles through a workspace and a
  // second launch) the selected inversion at ns = 1000, nt = 10 went from 58.8 to
  // 49.2 ms, at ns = 333, nt = 17 from 9.0 to 6.3.  64 is there for the fp64_tile knob.
  const int tm = g.tile == 64 ? 64 : 32, tk = tm == 64 ? 16 : 8;
  const double tiles = (double)tiles_written(g, tm) * g.batch;
  const ClusterRoom& room = cluster_room();
  int ksplit = 1;
  double best = 1e300;
  // beside the look-ahead stream's work the wide clusters of a product of many
  // tiles wait for room (factorization at ns = 1000, nt = 10 31.9 ms with up to 8,
  // 30.2 with up to 2); for few tiles the shorter launch still wins (ns = 333,
  // nt = 17 6.0 against 6.4)
  const int ks_max = g.beside && tiles > 76 ? 2 : 8;
  for (int ks = 1; ks <= ks_max; ++ks) {
    // a K step of the kernel a slice at least; nothing to gain past a few waves
    if (ks > 1 && (g.k < tk * ks || tiles > 8 * GB300_SMS || (long long)ks * g.batch > 65535)) break;
    double shares = std::ceil(tiles * ks / GB300_SMS);
    if (tiles > room.clusters[ks]) shares = std::max(shares, 2.0);
    const int part = ((g.k + ks - 1) / ks + tk - 1) / tk * tk;  // K terms of a slice
    const double us = shares * tm * tm * part / 3200.0 + (ks > 1 ? 2.0 : 0.0);
    if (us < best) {
      best = us;
      ksplit = ks;
    }
  }
  g.ksplit = ksplit;
  const dim3 grid((unsigned)tiles_written(g, tm), 1, ksplit * g.batch), cluster(1, 1, ksplit);
  if (tm == 32) launch_k_cluster(gemm_fp64_kernel<32, 8>, grid, dim3(128), cluster, 0, s, g);
  else launch_k_cluster(gemm_fp64_kernel<64, 16>, grid, dim3(128), cluster, 0, s, g);
  return 1;
}

void launch_trsm_rows(double* X, long long xrs, long long xcs, int rows, const double* L,
                      long long ldl, int nbk, int mode, int batch, long long sX, long long sL,
                      cudaStream_t s) {
  if (rows <= 0 || nbk <= 0 || batch <= 0) return;
  const bool wide = (long long)rows * batch <= 4 * GB300_SMS * 4;  // up to four CTAs of four rows an SM
  const dim3 grid((rows + (wide ? 3 : 15)) / (wide ? 4 : 16), batch);
  auto* kern = mode == 0 ? (wide ? trsm_rows_kernel<0, 32> : trsm_rows_kernel<0, 8>)
                         : (wide ? trsm_rows_kernel<1, 32> : trsm_rows_kernel<1, 8>);
  launch_k(kern, grid, dim3(128), 0, s, X, xrs, xcs, rows, L, ldl, nbk, sX, sL);
}

void launch_leaf_inverses(double* U, long long ldu, int n, const double* L, long long ldl,
                          int batch, long long sU, long long sL, cudaStream_t s) {
  if (n <= 0 || batch <= 0) return;
  const int leaves = (n + 63) / 64, rows = std::min(n, 64);
  const bool wide = (long long)rows * leaves * batch <= 4 * GB300_SMS * 4;
  const dim3 grid((rows + (wide ? 3 : 15)) / (wide ? 4 : 16), batch, leaves);
  launch_k(wide ? trsm_rows_kernel<0, 32, true> : trsm_rows_kernel<0, 8, true>, grid, dim3(128), 0, s,
           U, 1ll, ldu, rows, L, ldl, n, sU, sL);
}

}  // namespace rgf

// ---------------------------------------------------------------------------
// FP64 peak probe: independent DMMA m8n8k4 chains on every SM, used as the
// denominator of the FP64 roofline (the tensor-pipe FP64 rate of this GPU).
// ---------------------------------------------------------------------------
namespace rgf {
namespace {
__global__ void __launch_bounds__(256) dmma_peak_kernel(double* out, int iters) {
  double a = 1.0 + threadIdx.x * 1e-9, b = 0.5;
  double c[4][2] = {};
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) dmma_8x8x4(c[j], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) s += c[j][0] + c[j][1];
  out[(long long)blockIdx.x * blockDim.x + threadIdx.x] = s;
}
}  // namespace

int measure_fp64_peak(double* tflops) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 4;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 4;
  const int blocks = sms * 8, threads = 256, iters = 1024;
  double* buf = nullptr;
  if (cudaMalloc(&buf, sizeof(double) * blocks * threads) != cudaSuccess) return 2;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 3; ++rep) {
    cudaEventRecord(e0);
    dmma_peak_kernel<<<blocks, threads>>>(buf, iters);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0 && ms < best) best = ms;
  }
  cudaError_t err = cudaGetLastError();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(buf);
  if (err != cudaSuccess) return 4;
  const double flops = 2.0 * 8 * 8 * 4 * 4.0 * iters * (double)blocks * threads / 32.0;
  *tflops = flops / (best * 1e-3) / 1e12;
  return 0;
}
}  // namespace rgf
