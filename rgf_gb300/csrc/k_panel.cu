// FP64 kernels of the panel factorization: the Cholesky of a diagonal tile of
// up to 160 columns in one launch (a cluster of sixteen CTAs), and the triangular
// solve of the rows below it.
//
// On GB300 an FP64 warp instruction holds its SM sub-partition's FP64 unit ~76
// cycles (whatever the number of active lanes) and a dependent one waits ~65,
// so two things decide these kernels: the number of dependent FP64 operations
// per column (the pivot chain), and how many SMs share the FP64 work around it.
#include <algorithm>
#include <cstdint>

#include "rgf_device.h"
#include "rgf_internal.h"

namespace rgf {

namespace {

constexpr int LB = PANEL_LEAF;                 // leaf width: 32
constexpr int XPITCH = LB + 1;
constexpr int LEAF_WARPS = 8;                  // of the leaf CTA's warps; one more sends
constexpr int TILE_THREADS = (LEAF_WARPS + 1) * 32;

// d > 0 (and not NaN) by its bit pattern: an FP64 compare is an FP64 instruction
__device__ __forceinline__ bool positive_bits(double d) {
  const long long b = __double_as_longlong(d);
  return b > 0 && b <= 0x7ff0000000000000ll;
}

// 2 / m of a normal positive double d = m 2^e, m in [1, 2) (within 2^-62 relative before
// the final rounding) in integer arithmetic: no FP64 instruction on the pivot chain.
// y0 is an FP32 reciprocal of m's leading 24 bits (|1 - m y0| < 2^-22);
// with t = 1 - m y0 exact to 2^-62, one cubic step 1/m = y0 + y0 t + y0 t^2 leaves an
// error of t^3 < 2^-66.  Its dependent steps are single 32-bit operations and
// 32 x 32 -> 64 multiplications: ~150 cycles, where FP32 double-float refinement and
// two FP64 operations took ~230 and a reciprocal square root 454.
__device__ __forceinline__ double recip_significand(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;"
      : "=f"(y)
      : "f"(__uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u)));
  const unsigned Mh = __funnelshift_l(lo, hi, 11) | 0x80000000u, Ml = lo << 11;  // m 2^63
  // y0 2^32: y's significand (y in [0.5, 1]; 1 is taken as 1 - 2^-24)
  const unsigned Y0 = (min(__float_as_uint(y), 0x3f7fffffu) << 8) | 0x80000000u;
  const int Y31 = (int)(Y0 >> 1);
  const unsigned long long P = (unsigned long long)Mh * Y0 + __umulhi(Ml, Y0);  // m y0 2^63
  const long long E = (long long)(0x8000000000000000ull - P);                  // t 2^63
  const int Eh = (int)(E >> 20);                                               // t 2^43
  const int El = (int)(((unsigned)E & 0xfffffu) << 1);                         // rest, 2^64
  const int E2 = __mulhi((int)(E >> 10), Eh);                                  // t^2 2^64
  const long long A = (long long)Y31 * Eh;                                     // 2^74
  const long long D = (long long)Y31 * El + (long long)Y31 * E2;               // 2^95
  // 1/m 2^63 plus half a unit of the 53 bits kept
  const unsigned long long Y1 = (((unsigned long long)Y0 << 31) + 512) +
                                (unsigned long long)(A >> 11) +
                                (unsigned long long)(long long)(int)(D >> 32);
  return __longlong_as_double((long long)((1022ull << 52) + (Y1 >> 10)));
}
// the high word of 2^-(e + 1) less that of 1: added to another high word, it scales by it
__device__ __forceinline__ unsigned half_recip_power(double d) {
  return 0x3fe00000u - ((unsigned)__double2hiint(d) & 0x7ff00000u);
}

// x / d; NaN for a d that is not positive
__device__ __noinline__ double over_pivot_slow(double x, double d) {
  return positive_bits(d) ? x / d : __longlong_as_double(0x7ff8000000000000ll);
}
__device__ __forceinline__ double over_pivot(double x, double d) {
  const double r = recip_significand(d);
  // 1 / d has to be normal: 2^-1022 <= d < 2^1017
  if ((unsigned)__double2hiint(d) - 0x100000u >= 0x7f800000u) return over_pivot_slow(x, d);
  return x * __hiloint2double(__double2hiint(r) + (int)half_recip_power(d), __double2loint(r));
}
// a - v w / d.  The product of two entries of unscaled columns has the square of the
// matrix's magnitude, so w first gives up d's power of two (in its exponent field,
// beside the reciprocal): |v w / d| is at most that of a's row and column.  d and |w|
// between 2^-503 and 2^517 take that way (two range tests: every instruction of the
// leaf's loops counts); of the others a zero w has no term, the rest divide.
__device__ __forceinline__ double minus_term(double a, double v, double w, double d) {
  constexpr unsigned LO = 520u << 20, RANGE = 1020u << 20;
  const unsigned dh = (unsigned)__double2hiint(d), wh = (unsigned)__double2hiint(w);
  const double p = v * __hiloint2double((int)(wh + half_recip_power(d)), __double2loint(w));
  double x = fma(-p, recip_significand(d), a);
  asm volatile("" : "+d"(x));  // the rare branch stands behind the chain, not in it
  if (max(dh - LO, (wh & 0x7fffffffu) - LO) >= RANGE) {
    const bool no_term = dh - LO < RANGE && ((wh << 1) | (unsigned)__double2loint(w)) == 0 &&
                         ((unsigned)__double2hiint(v) & 0x7fffffffu) < 0x7ff00000u;
    x = a;
    if (!no_term) x = fma(-v, over_pivot_slow(w, d), a);
  }
  return x;
}

// ---- hand-off of doubles through shared memory -----------------------------------
// A slot holds UNSET until its value is stored; the reader polls the slot
// itself, so no flag, fence or barrier stands between producer and consumer
// (a release / acquire flag costs ~85 cycles more).  UNSET is a NaN recognized
// by its high word; a value with that high word (a NaN) is stored as the
// canonical NaN.  Polls are bounded by `polls` (the bound is the only thing a poll loop
// counts: it has to turn around in a few cycles); one that runs out records a
// timeout and sets abort_, after which the CTA's later leaves are skipped and a
// thread's later polls in the same leaf end at once.  abort_ may be set at any
// time by a warp whose own wait ran out, so whatever stands before a barrier
// is decided from one reduction over all the barrier's threads (bar_any_leaf within
// a leaf, __syncthreads_or after it), never from a warp's own read.
constexpr int UNSET_HI = 0x7ff85e5e;
constexpr unsigned long long CANON_NAN = 0x7ff8000000000000ull;

struct Wait {
  volatile int* abort_;
  DevStatus* st;
  int polls;
};

__device__ __forceinline__ bool slot_empty(double v) { return __double2hiint(v) == UNSET_HI; }
__device__ __forceinline__ double slot_clean(double v) {
  return slot_empty(v) ? __longlong_as_double((long long)CANON_NAN) : v;
}
// a wait ran out
__device__ __noinline__ void wait_gave_up(const Wait& w) {
  atomicExch(&w.st->timeout, 1);
  *w.abort_ = 1;
}
// Slots by their 32-bit shared-memory address: the leaf's loops run one warp per
// scheduler, so every instruction counts.
__device__ __forceinline__ double lds_peek(unsigned addr) {
  double v;
  asm volatile("ld.volatile.shared::cta.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts_slot(unsigned addr, double v) {
  asm volatile("st.volatile.shared::cta.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ double lds_wait(unsigned addr, const Wait& w, bool& over) {
  double v = lds_peek(addr);
  int left = over ? 0 : w.polls;
#pragma unroll 1
  while (slot_empty(v)) {
    if (--left <= 0) {
      over = true;
      break;
    }
    v = lds_peek(addr);
  }
  return v;
}

// ---- leaf: A = V D^-1 V^T of a <= 32 x 32 tile in one CTA of four warps ----------
// Square-root free: column j is published unscaled (V_rj, with V_jj = d_j the
// pivot), later its unit form l_rj = V_rj / d_j.  Columns take a_rc -= V_rj l_cj;
// the column that comes next takes a_rc - (V_rj V_cj) (1 / d_j) instead, from V
// alone: its warp forms the product and the reciprocal side by side (d_j's power of
// two is taken out of V_cj before the product, by its exponent field: the product
// itself would leave FP64's range for entries past 1e+-154).  So the
// chain per column is one hand-off, the reciprocal and one FMA (~400 cycles, 500
// with the warps that come late; a second hand-off, of the reciprocal, made it
// 560-650).  The columns become
// L_rj = V_rj d_j^{-1/2} once, at the end, off the chain.
// The columns go in two halves of 16; between them the trailing 16 x 16 block
// takes the first half's terms with one element a thread.  (A column's FMA of 32
// row lanes costs the same whatever rows are live: right-looking over all 32
// columns is 496 of them, this is 240 + 68.)  Within a half, column c lives in a
// register of warp c % 8, lane = row; a warp brings its first column up to date
// and publishes it before it turns to its second one, in one small loop body
// (the code has to stay in the instruction cache).  Two columns a warp leave a
// warp ~200 cycles of work per step, below the chain; with four, the warps were
// late and set the pace (~650 cycles a column).  A ninth warp sends the unit
// columns to the workers as they appear and takes the square roots.
// A 32-column leaf takes ~11 us (21 K cycles, hand-off to the workers included);
// the previous one, with reciprocal square roots and column flags, 20.7 us.
struct LeafShared {
  int abort_, fail;
};

// columns [b0, b1) of the leaf, already updated by the columns before b0 (the leaf warps)
__device__ __forceinline__ void leaf_half(const double (*S)[LB], double (*V)[LB], double (*Lc)[LB],
                                          int b0, int b1, int nbk, LeafShared* sh, const Wait& w) {
  static_assert(LEAF_WARPS * 2 == LB / 2, "two columns a warp");
  constexpr int ROW = LB * sizeof(double);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned sv = (unsigned)__cvta_generic_to_shared(V) + lane * 8;
  const unsigned sl = (unsigned)__cvta_generic_to_shared(Lc);
  auto first = [&](int c) { return c < b1 && lane >= c && lane < nbk ? S[c][lane] : 0.0; };
  bool over = false;
  // a -= column j times column c's multiplier l_cj
  auto step = [&](double a, int j, int c) {
    double l, v;
    int left = over ? 0 : w.polls;
#pragma unroll 1
    for (;;) {
      l = lds_peek(sl + j * ROW + c * 8);
      v = lds_peek(sv + j * ROW);  // published before l
      if (!(slot_empty(l) | slot_empty(v))) break;
      if (--left <= 0) {
        over = true;
        break;
      }
    }
    __syncwarp();
    return fma(-v, l, a);
  };
  double a = first(b0 + warp);
#pragma unroll 1
  for (int c = b0 + warp; c < b1; c += LEAF_WARPS) {
    int j = b0;
#pragma unroll 1
    for (; j + 1 < c; ++j) a = step(a, j, c);
    if (c > b0) {  // the last step, from column j alone
      const double v = lds_wait(sv + j * ROW, w, over);
      __syncwarp();
      a = minus_term(a, v, __shfl_sync(0xffffffffu, v, c), __shfl_sync(0xffffffffu, v, j));
    }
    a = slot_clean(a);
    sts_slot(sv + c * ROW, a);
    const double d = __shfl_sync(0xffffffffu, a, c);
    const double l = over_pivot(a, d);
    sts_slot(sl + c * ROW + lane * 8, lane > c ? slot_clean(l) : 0.0);
    if (lane == 0 && !positive_bits(d)) atomicMin(&sh->fail, c);
    if (__any_sync(0xffffffffu, over)) {
      if (lane == 0) wait_gave_up(w);
      return;
    }
    a = first(c + LEAF_WARPS);
  }
}

// barrier of the leaf warps
__device__ __forceinline__ void bar_sync_leaf() {
  asm volatile("bar.sync 1, %0;" ::"n"(LEAF_WARPS * 32) : "memory");
}
// the same; whether any of their threads brought `stop`: all of them get one answer
__device__ __forceinline__ bool bar_any_leaf(bool stop) {
  int any;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n"
      " selp.s32 %0, 1, 0, q;\n}"
      : "=r"(any) : "r"((int)stop), "n"(LEAF_WARPS * 32) : "memory");
  return any != 0;
}

// S(r, c) -= sum_{j < 16} V_rj l_cj over the lower elements 16 <= c <= r < 32 of the
// second half (136 of them; the terms are summed before they meet S, here and in
// all updates between leaves, so that S's size rounds once a leaf and not once a
// column: at ns = 128 that is 1.4 times less error in the factor): two neighbouring threads share an element's 16
// terms, and the last eight elements go to one warp, four threads each
__device__ __forceinline__ void leaf_trailing(double (*S)[LB], const double (*V)[LB],
                                              const double (*Lc)[LB]) {
  constexpr int H = LB / 2;
  auto element = [](int e, int& r, int& c) {  // e = r' (r' + 1) / 2 + c', r' = r - 16
    r = (int)((sqrtf((float)(8 * e + 1)) - 1.0f) * 0.5f);  // exact for e < 136
    c = e - r * (r + 1) / 2 + H;
    r += H;
  };
  const int t = threadIdx.x;
  int r, c;
  element(t >> 1, r, c);
  int j0 = (t & 1) * (H / 2);
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < H / 2; ++j) s = fma(V[j0 + j][r], Lc[j0 + j][c], s);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  if ((t & 1) == 0) S[c][r] -= s;
  if (t >= LEAF_WARPS * 32 - 32) {
    element(LEAF_WARPS * 16 + ((t & 31) >> 2), r, c);
    j0 = (t & 3) * (H / 4);
    s = 0.0;
#pragma unroll
    for (int j = 0; j < H / 4; ++j) s = fma(V[j0 + j][r], Lc[j0 + j][c], s);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((t & 3) == 0) S[c][r] -= s;
  }
}

__device__ __forceinline__ void leaf_ldl(double (*S)[LB], double (*V)[LB], double (*Lc)[LB],
                                         int nbk, LeafShared* sh, const Wait& w) {
#pragma unroll 1
  for (int b0 = 0; b0 < nbk; b0 += LB / 2) {
    if (b0 > 0) {
      if (bar_any_leaf(*w.abort_ != 0)) return;
      leaf_trailing(S, V, Lc);
      bar_sync_leaf();
    }
    leaf_half(S, V, Lc, b0, min(b0 + LB / 2, nbk), nbk, sh, w);
  }
}

// The leaf CTA's last warp: sends every unit column to the workers (push) as it
// appears, then takes d^{-1/2} of all pivots and sends those too.
template <int NW>
__device__ __forceinline__ void leaf_send(const double (*V)[LB], const double (*Lc)[LB], double* ys,
                                          int nbk, const Wait& w, bool push) {
  const int lane = threadIdx.x & 31;
  bool over = false;
  auto send = [&](const double* p, double v) {
#pragma unroll 3
    for (int q = 1; q <= NW; ++q) st_cluster(cluster_addr(p, q), v);
  };
  auto send_column = [&](int c) {
    const double l = lds_wait((unsigned)__cvta_generic_to_shared(&Lc[c][lane]), w, over);
    __syncwarp();
    send(&Lc[c][lane], l);
  };
  if (push) {
#pragma unroll 1
    for (int c = 0; c + 1 < nbk && !__any_sync(0xffffffffu, over); ++c) send_column(c);
  }
  const double d =
      lane < nbk ? lds_wait((unsigned)__cvta_generic_to_shared(&V[lane][lane]), w, over) : 1.0;
  __syncwarp();
  const double y = positive_bits(d) ? rsqrt_fast(d) : __longlong_as_double((long long)CANON_NAN);
  ys[lane] = y;
  if (push) {
    send_column(nbk - 1);
    send(&ys[lane], y);
  }
  if (__any_sync(0xffffffffu, over) && lane == 0) wait_gave_up(w);
}

// In-block part of x L^T = b for one row against a leaf, z-form: lane q of the
// row's G lanes holds columns t G + q in u[t]; on return u holds z (x before
// the scaling by d^{-1/2}).  Only FMAs whose slot can hold a live column are
// issued.  STREAM: the unit columns are polled as the leaf publishes them.
template <int G, bool STREAM>
__device__ __forceinline__ void leaf_row_solve(double (&u)[LB / G], const double (*Lc)[LB],
                                               int nbk, int lane, const Wait& w, bool& over) {
  const int q = lane & (G - 1), gbase = lane & ~(G - 1);
  const unsigned sl = (unsigned)__cvta_generic_to_shared(Lc) + q * 8;
#pragma unroll
  for (int t = 0; t < LB / G; ++t) {
#pragma unroll 1
    for (int jj = 0; jj < G; ++jj) {
      const int j = t * G + jj;
      if (j >= nbk) return;
      double l[LB / G];
      if (STREAM) {
        int left = w.polls;
#pragma unroll 1
        for (;;) {
          bool e = false;
#pragma unroll
          for (int s = t; s < LB / G; ++s) {
            l[s] = lds_peek(sl + (j * LB + s * G) * 8);
            e |= slot_empty(l[s]);
          }
          if (!e) break;
          if (--left <= 0) {
            over = true;
            break;
          }
        }
        if (__any_sync(0xffffffffu, over)) return;
      } else {
#pragma unroll
        for (int s = t; s < LB / G; ++s) l[s] = Lc[j][s * G + q];
      }
      const double z = -__shfl_sync(0xffffffffu, u[t], gbase | jj);
      const double nv = fma(z, l[t], u[t]);
      u[t] = q > jj ? nv : u[t];
#pragma unroll
      for (int s = t + 1; s < LB / G; ++s) u[s] = fma(z, l[s], u[s]);
    }
  }
}

// ---- the tile: Cholesky of the w x w (w <= 160) lower tile at P ----------------
// Rank 0 (the leaf CTA) factors the 32-wide leaves one after another; NW
// workers hold the tile's other rows (row 32 + rank - 1 + NW i each) in shared
// memory.  Step k:
//   the leaf CTA factors leaf k, sending its unit columns as they appear;
//   the workers solve their rows against them one column behind (WG lanes a
//   row), write the result to P and send the next leaf block's rows to each other
//   -- cluster barrier --
//   the workers update the elements of the next leaf and send them to the leaf CTA
//   -- cluster barrier (split: the leaf CTA goes on, the workers first update
//      the rest of their rows behind the next leaf's chain) --
// P is read by the workers' non-critical updates through L2.  Fifteen workers
// keep those updates shorter than the leaf's chain (seven are ~5 us late once per
// 128-wide tile).  Shared memory stays below 28 KiB and registers at 40 a
// thread, so that the CTAs fit beside the split GEMM's (198 KiB, 54 K registers)
// that the side stream runs meanwhile.  The unit leaves and d^{-1/2} also go to
// ws (PANEL_WS doubles) for panel_rows_kernel.
// Measured: 57 us for a 128-column tile, where four leaf launches (29 us each)
// with their row solves (15 us) and three small products took ~215 us;
// factorization of ns = 128, nt = 10 in split precision 1.86 -> 0.88 ms, of
// ns = 2000, nt = 4 17.1 -> 13.2 ms (11.7 ms launched directly).
template <int NW, int TW>  // workers; widest tile
__global__ void __launch_bounds__(TILE_THREADS, 5)
    panel_tile_kernel(double* P, long long lda, int w, double* ws, int col0, DevStatus* st,
                      int wait_polls) {
  constexpr int WROWS = (TW - LB + NW - 1) / NW;  // tile rows of one worker
  constexpr int WG = WROWS > 8 ? 16 : 32;         // lanes a row in the workers' solve
  // a worker's rows, packed: at most WROWS rows, the longest of them TW
  constexpr int OWN = WROWS * TW - NW * (WROWS * (WROWS - 1) / 2);
  __shared__ __align__(16) double Lc[LB][LB];     // unit columns of the current leaf
  __shared__ double ys[LB];                       // d^{-1/2}
  // leaf CTA: S | V; workers: packed own rows | x of the next leaf block
  __shared__ double bufA[OWN > LB * LB ? OWN : LB * LB];
  __shared__ double bufB[LB * XPITCH];
  __shared__ LeafShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nl = (w + LB - 1) / LB;
  const int rank = blockIdx.x;  // the grid is one cluster (one CTA when nl == 1)
  const double unset = __hiloint2double(UNSET_HI, 0);
  const Wait wait{&sh.abort_, st, wait_polls};
  auto clear_slots = [&]() {  // Lc and ys before the next leaf
    for (int e = tid; e < LB * LB; e += TILE_THREADS) (&Lc[0][0])[e] = unset;
    if (tid < LB) ys[tid] = unset;
  };
  clear_slots();
  if (tid == 0) {
    sh.abort_ = 0;
    sh.fail = 0x7fffffff;
  }
  pdl_wait();
  if (rank == 0) {
    double(*S)[LB] = reinterpret_cast<double(*)[LB]>(bufA);
    double(*V)[LB] = reinterpret_cast<double(*)[LB]>(bufB);
    for (int c = warp; c < min(LB, w); c += TILE_THREADS / 32)
      if (lane >= c && lane < w) S[c][lane] = P[lane + (long long)c * lda];
    for (int e = tid; e < LB * LB; e += TILE_THREADS) bufB[e] = unset;
    __syncthreads();
    if (nl > 1) { cluster_arrive(); cluster_wait(); }
    bool stop = false;
    for (int k = 0; k < nl; ++k) {
      const int nbk = min(LB, w - k * LB);
      if (!stop) {
        if (warp < LEAF_WARPS) leaf_ldl(S, V, Lc, nbk, &sh, wait);
        else leaf_send<NW>(V, Lc, ys, nbk, wait, k + 1 < nl);
      }
      stop = __syncthreads_or(*wait.abort_);
      if (k + 1 < nl) cluster_arrive();  // (workers: rows solved)
      else pdl_trigger();                // the next kernel's CTAs may come in
      // results: L = V d^{-1/2} to P, the unit columns and d^{-1/2} to ws
      double* D = P + (long long)k * LB * (lda + 1);
      double* W = ws + (long long)k * PANEL_LEAF_WS;
      for (int c = warp; c < LB; c += TILE_THREADS / 32) {
        const bool in = c < nbk && lane < nbk;
        if (in && lane >= c) D[lane + (long long)c * lda] = V[c][lane] * ys[c];
        W[c * LB + lane] = in && lane > c ? Lc[c][lane] : 0.0;
      }
      if (warp == 0) W[LB * LB + lane] = lane < nbk ? ys[lane] : 0.0;
      if (tid == 0) {
        if (sh.fail != 0x7fffffff) atomicMin(&st->not_spd_col, col0 + k * LB + sh.fail);
        sh.fail = 0x7fffffff;
      }
      if (k + 1 == nl) break;
      __syncthreads();
      clear_slots();
      for (int e = tid; e < LB * LB; e += TILE_THREADS) bufB[e] = unset;
      __syncthreads();
      cluster_wait();
      cluster_arrive();  // (workers: next leaf in S)
      cluster_wait();
    }
    return;
  }

  // ---- workers ----
  const int row0 = LB + rank - 1;                 // own row i: row0 + NW i
  const int nown = w > row0 ? (w - row0 + NW - 1) / NW : 0;
  auto own = [&](int i) -> double* { return bufA + i * (row0 + 1) + NW * (i * (i - 1) / 2); };
  double(*Xn)[XPITCH] = reinterpret_cast<double(*)[XPITCH]>(bufB);
  for (int i = warp; i < nown; i += TILE_THREADS / 32) {
    const int r = row0 + NW * i;
    for (int c = lane; c <= r; c += 32) own(i)[c] = P[r + (long long)c * lda];
  }
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  bool stop = false;
  for (int k = 0; k + 1 < nl; ++k) {
    const int kc = k * LB, kn = kc + LB;          // this leaf's and the next one's first column
    {  // solve: WG lanes a row, ROUND rows at a time
      constexpr int SL = LB / WG, ROUND = LEAF_WARPS * (32 / WG);
      const int q = lane & (WG - 1);
      bool over = false;
#pragma unroll 1
      for (int i0 = 0; i0 < WROWS && warp < LEAF_WARPS && !stop; i0 += ROUND) {
        const int i = i0 + warp * (32 / WG) + lane / WG;
        const int r = row0 + NW * i;
        const bool live = i < nown && r >= kn;
        if (!__any_sync(0xffffffffu, live)) continue;
        double u[SL];
#pragma unroll
        for (int t = 0; t < SL; ++t) u[t] = live ? own(i)[kc + t * WG + q] : 0.0;
        leaf_row_solve<WG, true>(u, Lc, LB, lane, wait, over);
#pragma unroll
        for (int t = 0; t < SL; ++t) {
          const int c = t * WG + q;
          const double x =
              u[t] * lds_wait((unsigned)__cvta_generic_to_shared(&ys[c]), wait, over);
          if (live) {
            if (r < kn + LB) {
#pragma unroll
              for (int z = 1; z <= NW; ++z) st_cluster(cluster_addr(&Xn[r - kn][c], z), x);
            }
            own(i)[kc + c] = x;
            P[r + (long long)(kc + c) * lda] = x;
          }
        }
        if (__any_sync(0xffffffffu, over)) {
          if (lane == 0) wait_gave_up(wait);
          break;
        }
      }
    }
    stop = __syncthreads_or(*wait.abort_);
    clear_slots();
    __syncthreads();
    cluster_arrive();
    cluster_wait();                               // every row is solved
    // next leaf: own rows r in [kn, kn + 32), columns kn..r; KS neighbouring threads
    // share an element's 32 terms
    {
      constexpr int KS = NW >= 15 ? 4 : 2;        // at most 256 / KS elements
      int e = tid / KS, i = (max(kn - row0, 0) + NW - 1) / NW, r = row0 + NW * i;
      while (i < nown && r < kn + LB && e > r - kn) {
        e -= r - kn + 1;
        ++i;
        r += NW;
      }
      const bool live = i < nown && r < kn + LB;  // element (r, kn + e)
      if (__any_sync(0xffffffffu, live)) {
        const int l0 = (tid % KS) * (LB / KS);
        double s = 0.0;
        const double* xr = Xn[live ? r - kn : 0] + l0;
        const double* xc = Xn[live ? e : 0] + l0;
#pragma unroll
        for (int l = 0; l < LB / KS; ++l) s = fma(xr[l], xc[l], s);
#pragma unroll
        for (int o = 1; o < KS; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (live && l0 == 0)
          st_cluster(cluster_addr(bufA + e * LB + (r - kn), 0), own(i)[kn + e] - s);
      }
    }
    __syncthreads();
    cluster_arrive();                             // the leaf CTA may go on
    // the rest: own rows past the next leaf, columns kn..r, 32 columns a unit
    {
      int unit = 0;
      for (int i = (max(kn + LB - row0, 0) + NW - 1) / NW; i < nown; ++i) {
        const int r = row0 + NW * i;
        for (int c0 = kn; c0 <= r; c0 += LB, ++unit) {
          if (unit % (TILE_THREADS / 32) != warp) continue;
          const int c = c0 + lane;
          const bool live = c <= r;
          const double* xc = P + (live ? c : r) + (long long)kc * lda;
          const double* xr = own(i) + kc;
          double s = 0.0;
#pragma unroll 1
          for (int l0 = 0; l0 < LB; l0 += 8) {
            double b[8];
#pragma unroll
            for (int l = 0; l < 8; ++l) {
              b[l] = __ldcg(xc);
              xc += lda;
            }
#pragma unroll
            for (int l = 0; l < 8; ++l) s = fma(xr[l0 + l], b[l], s);
          }
          if (live) own(i)[c] -= s;
        }
      }
    }
    __syncthreads();
    cluster_wait();
  }
  pdl_trigger();
}

// ---- rows below the tile: X := X L^{-T} for `rows` rows of w columns -------------
// Bound by the FP64 units (w^2 / 2 FMAs a row).  G lanes share a row, lane q of
// them holds columns t G + q in registers, and a CTA of four warps takes 128 / G
// rows: G is chosen so that the rows cover the SMs once (launch_panel_rows).
// Per 32-column block k: the unit leaf (from ws) solves the block (z-form), the
// scaled result updates the columns after it with the tile's rows of block k.
// The leaf and the rows of the block are copied to shared memory asynchronously,
// the latter (and the next leaf) behind the solve.
template <int G, int NB, int NT>  // NB: 32-column blocks of the tile (the last may be narrower)
__global__ void __launch_bounds__(NT)
    panel_rows_kernel(double* X, int rows, const double* P, long long lda, int w,
                      const double* ws) {
  constexpr int SB = LB / G;        // register slots of one block
  constexpr int XR = (NB - 1) * LB; // tile rows below the first leaf
  __shared__ __align__(16) double Lc[LB][LB];
  __shared__ double ys[LB];
  __shared__ double Xs[XR > 0 ? LB : 1][XR > 0 ? XR : 1];  // [l][c - 32 (k + 1)]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q = lane & (G - 1), gbase = lane & ~(G - 1);
  const int row = blockIdx.x * (NT / G) + warp * (32 / G) + lane / G;
  const bool live = row < rows;
  pdl_wait();
  auto fetch_leaf = [&](int k) {
    const double* W = ws + (long long)k * PANEL_LEAF_WS;
    for (int e = tid; e < LB * LB; e += NT) cp_async8(&Lc[0][0] + e, W + e);
    if (tid < LB) cp_async8(&ys[tid], W + LB * LB + tid);
    cp_async_commit();
  };
  fetch_leaf(0);
  double u[NB * SB];
#pragma unroll
  for (int t = 0; t < NB * SB; ++t) {
    const int c = t * G + q;
    u[t] = live && c < w ? X[row + (long long)c * lda] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    const int kc = k * LB, kn = kc + LB;
    if (k + 1 < NB) {
      const double* src = P + kn + (long long)kc * lda;
      for (int l = warp; l < LB; l += NT / 32)
        for (int c = lane; c < w - kn; c += 32) cp_async8(&Xs[l][c], src + c + (long long)l * lda);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    double z[SB];
#pragma unroll
    for (int t = 0; t < SB; ++t) z[t] = u[k * SB + t];
    bool over = false;
    leaf_row_solve<G, false>(z, Lc, min(LB, w - kc), lane, Wait{}, over);
#pragma unroll
    for (int t = 0; t < SB; ++t) u[k * SB + t] = z[t] * ys[t * G + q];
    if (k + 1 < NB) {
      cp_async_wait<0>();
      __syncthreads();
      fetch_leaf(k + 1);
      double sum[NB * SB];  // of this block's terms, before they meet u
#pragma unroll
      for (int s = (k + 1) * SB; s < NB * SB; ++s) sum[s] = 0.0;
#pragma unroll
      for (int t = 0; t < SB; ++t) {
#pragma unroll 1
        for (int jj = 0; jj < G; ++jj) {
          const double x = __shfl_sync(0xffffffffu, u[k * SB + t], gbase | jj);
          const double* xr = &Xs[t * G + jj][q];
#pragma unroll
          for (int s = (k + 1) * SB; s < NB * SB; ++s)
            sum[s] = fma(x, xr[s * G - kn], sum[s]);
        }
      }
#pragma unroll
      for (int s = (k + 1) * SB; s < NB * SB; ++s) u[s] -= sum[s];
      __syncthreads();  // Xs is overwritten next
    }
  }
  pdl_trigger();
  if (live) {
#pragma unroll
    for (int t = 0; t < NB * SB; ++t) {
      const int c = t * G + q;
      if (c < w) X[row + (long long)c * lda] = u[t];
    }
  }
}

// ---- chain: all block columns of a matrix of small blocks in one launch ----------
// For ns <= 64 (one or two leaves a block) the launches of a block (tile, rows, update of
// the next block) cost more than their work.  One cluster walks the block columns.
// Every CTA holds the current diagonal leaf and factors it itself (its ~11 us a 32
// columns are a serial chain: doing it NC times over costs nothing and saves sending
// it); the other rows of the block column (rows 32.. of the diagonal block, then the nd
// arrowhead rows, then the rows of the block below: row t at CTA t % NC) are solved
// behind the leaf by the CTA that owns them, in shared memory, and go to all CTAs.
// Then each CTA computes its share of the next leaf (or, after the last leaf, of the
// next block: its leaf by elements, its rows by owner) and sends the leaf's elements to
// all.  Two cluster barriers a leaf; the next block column's entries come by
// asynchronous copies meanwhile.
// The leaf's pivot chain bounds it (~0.35 us a column, of ~0.45 in all).  Factorization
// of 40 blocks, launches per block -> this: ns = 3 0.35 -> 0.21 ms, ns = 16 0.64 -> 0.37,
// ns = 32 0.90 -> 0.59, ns = 42 1.34 -> 0.87, ns = 64 1.61 -> 1.28 (0.13 ms of each the
// ingest, the corner and the log-determinant).
constexpr int CHAIN_ROW_WARPS = 8;
constexpr int CHAIN_THREADS = TILE_THREADS + CHAIN_ROW_WARPS * 32;  // leaf, d^{-1/2}, rows

struct ChainShape {  // of one CTA's shared memory
  int nD, rows, pitch;
  __host__ __device__ ChainShape(int ns, int nd, int nc)
      : nD(ns > LB ? ns - LB : 0), rows((nD + nd + ns + nc - 1) / nc), pitch(ns | 1) {}
  // own rows twice | rows of the block below | rows 32.. of the diagonal block | own
  // elements of the next block's leaf
  __host__ __device__ size_t elems(int ns, int nc) const {
    return 2 * (size_t)rows * pitch + (size_t)ns * pitch + (size_t)nD * XPITCH +
           (LB * (LB + 1) / 2 + nc - 1) / nc;
  }
};

__global__ void __launch_bounds__(CHAIN_THREADS, 1)
    chain_factor_kernel(double* MF, int ns, int nd, long long nt, DevStatus* st, int wait_polls) {
  extern __shared__ double dyn[];
  __shared__ __align__(16) double Lc[LB][LB];
  __shared__ double S[LB][LB], V[LB][LB], ys[LB];
  __shared__ LeafShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nc = gridDim.x, rank = blockIdx.x;
  const ChainShape z(ns, nd, nc);
  const int nD = z.nD, nl = nD ? 2 : 1, xp = z.pitch, n0 = min(ns, LB);
  double* X0 = dyn;                                  // own row j: t = rank + nc j
  double* XB = X0 + 2 * z.rows * xp;                 // solved rows of the block below
  double(*XD)[XPITCH] = reinterpret_cast<double(*)[XPITCH]>(XB + ns * xp);
  double* E = XB + ns * xp + nD * XPITCH;            // element rank + nc e of the next leaf
  const int leaf_elems = n0 * (n0 + 1) / 2;
  const int ne = leaf_elems > rank ? (leaf_elems - rank + nc - 1) / nc : 0;
  const double unset = __hiloint2double(UNSET_HI, 0);
  const Wait wait{&sh.abort_, st, wait_polls};
  auto clear_slots = [&]() {
    for (int e = tid; e < LB * LB; e += CHAIN_THREADS) (&Lc[0][0])[e] = (&V[0][0])[e] = unset;
    if (tid < LB) ys[tid] = unset;
  };
  auto element = [](int x, int& r, int& c) {         // x = r (r + 1) / 2 + c
    r = (int)((sqrtf((float)(8 * x + 1)) - 1.0f) * 0.5f);  // exact for x < 528
    c = x - r * (r + 1) / 2;
  };
  const long long sP = (long long)ns * (2 * ns + nd);
  auto rows_of = [&](long long i) {                  // own rows in block column i
    const int all = nD + nd + (i < nt - 1 ? ns : 0);
    return all > rank ? (all - rank + nc - 1) / nc : 0;
  };
  // row t of block column i within its panel
  auto row_at = [&](int t, bool last) {
    return t < nD ? LB + t : t < nD + nd ? (last ? ns : 2 * ns) + t - nD : ns + t - nD - nd;
  };
  auto fetch_rows = [&](long long i) {
    const bool last = i == nt - 1;
    const double* P = MF + i * sP;
    const long long lda = (last ? ns : 2 * ns) + nd;
    double* X = X0 + (i & 1) * z.rows * xp;
    const int n = rows_of(i);
    for (int j = warp; j < n; j += CHAIN_THREADS / 32) {
      const int t = rank + nc * j, r = row_at(t, last), len = t < nD ? LB + t + 1 : ns;
      for (int c = lane; c < len; c += 32) cp_async8(X + j * xp + c, P + r + c * lda);
    }
  };
  clear_slots();
  if (tid == 0) {
    sh.abort_ = 0;
    sh.fail = 0x7fffffff;
  }
  pdl_wait();
  fetch_rows(0);
  cp_async_commit();
  {
    const long long lda = (nt == 1 ? ns : 2 * ns) + nd;
    for (int c = warp; c < n0; c += CHAIN_THREADS / 32)
      if (lane >= c && lane < n0) S[c][lane] = MF[lane + c * lda];
  }
  cp_async_wait<0>();
  __syncthreads();
  cluster_sync();  // every CTA is here before the first remote store

  bool stop = false;
  for (long long i = 0; i < nt; ++i) {
    const bool last = i == nt - 1;
    double* P = MF + i * sP;
    const long long lda = (last ? ns : 2 * ns) + nd;
    double* X = X0 + (i & 1) * z.rows * xp;
    double* Xn = X0 + ((i + 1) & 1) * z.rows * xp;
    const int nown = rows_of(i);
    if (!last) {  // the next block column: own rows, own elements of its leaf
      fetch_rows(i + 1);
      const double* Pn = P + sP;
      const long long ldn = (i + 1 == nt - 1 ? ns : 2 * ns) + nd;
      for (int e = tid; e < ne; e += CHAIN_THREADS) {
        int r, c;
        element(rank + nc * e, r, c);
        cp_async8(E + e, Pn + r + c * ldn);
      }
    }
    cp_async_commit();
#pragma unroll 1
    for (int k = 0; k < nl; ++k) {
      const int kc = k * LB, nbk = min(LB, ns - kc);
      if (!stop) {
        if (warp < LEAF_WARPS) {
          leaf_ldl(S, V, Lc, nbk, &sh, wait);
        } else if (warp == LEAF_WARPS) {
          leaf_send<1>(V, Lc, ys, nbk, wait, false);
        } else {
          constexpr int WG = 16, SL = LB / WG;       // two rows a warp
          const int q = lane & (WG - 1);
#pragma unroll 1
          for (int j0 = (warp - LEAF_WARPS - 1) * 2; j0 < nown; j0 += CHAIN_ROW_WARPS * 2) {
            const int j = j0 + lane / WG, t = rank + nc * j;
            const bool live = j < nown && (k == 0 || t >= nD);
            if (!__any_sync(0xffffffffu, live)) continue;
            bool over = false;
            double u[SL];
#pragma unroll
            for (int s = 0; s < SL; ++s) {
              const int c = s * WG + q;
              u[s] = live && c < nbk ? X[j * xp + kc + c] : 0.0;
            }
            leaf_row_solve<WG, true>(u, Lc, nbk, lane, wait, over);
            const int r = row_at(t, last);
#pragma unroll
            for (int s = 0; s < SL; ++s) {
              const int c = s * WG + q;
              const double x =
                  u[s] * lds_wait((unsigned)__cvta_generic_to_shared(&ys[c]), wait, over);
              if (live && c < nbk) {
                X[j * xp + kc + c] = x;
                P[r + (kc + c) * lda] = x;
                double* all = t < nD ? &XD[t][c]
                              : t >= nD + nd ? XB + (t - nD - nd) * xp + kc + c : nullptr;
                if (all)
                  for (int w = 0; w < nc; ++w) st_cluster(cluster_addr(all, w), x);
              }
            }
            if (__any_sync(0xffffffffu, over)) {
              if (lane == 0) wait_gave_up(wait);
              break;
            }
          }
        }
      }
      stop = __syncthreads_or(*wait.abort_);
      cluster_arrive();
      // L = V d^{-1/2}: each CTA writes its share of the leaf's columns
      for (int c = rank + nc * warp; c < nbk; c += nc * (CHAIN_THREADS / 32))
        if (lane >= c && lane < nbk)
          P[kc + lane + (kc + c) * lda] = V[c][lane] * ys[c];
      if (tid == 0) {
        if (rank == 0 && sh.fail != 0x7fffffff)
          atomicMin(&st->not_spd_col, (int)(i * ns) + kc + sh.fail);
        sh.fail = 0x7fffffff;
      }
      cp_async_wait<0>();
      __syncthreads();
      clear_slots();
      __syncwarp();
      cluster_wait();                                // every row is solved
      if (k + 1 == nl && last) break;
      // updates: element e of this CTA is init - a . b over `terms` terms
      const bool schur = k + 1 == nl;
      const int terms = schur ? ns : LB;
      int n = schur ? ne : 0;
      auto row_len = [&](int j) {                    // elements of own row j
        const int t = rank + nc * j;
        if (schur) return t < nD ? LB + t + 1 : t < nD + nd ? ns : 0;
        return t < nD ? t + 1 : nD;
      };
      for (int j = 0; j < nown; ++j) n += row_len(j);
      int ks = 1;
      {
        int cost = 1 << 30;
        for (int w = 1, lg = 1; w <= 8; w *= 2, ++lg) {
          const int rounds = (n * w + CHAIN_THREADS - 1) / CHAIN_THREADS;
          const int x = rounds * ((terms + w - 1) / w + lg);
          if (x < cost) {
            cost = x;
            ks = w;
          }
        }
      }
      const int t8 = tid & (ks - 1);
#pragma unroll 1
      for (int e0 = 0; e0 < n; e0 += CHAIN_THREADS / ks) {
        int e = e0 + tid / ks;
        const bool live = e < n;
        if (!__any_sync(0xffffffffu, live)) continue;
        if (!live) e = 0;
        double *dst, init;
        const double *a, *b;
        bool all;
        if (schur && e < ne) {
          int r, c;
          element(rank + nc * e, r, c);
          a = XB + r * xp;
          b = XB + c * xp;
          init = E[e];
          dst = &S[c][r];
          all = true;
        } else {
          if (schur) e -= ne;
          int j = 0;
          while (e >= row_len(j)) e -= row_len(j++);
          const int t = rank + nc * j;
          all = !schur && t < nD;
          a = schur && t < nD ? XB + (LB + t) * xp : X + j * xp;
          b = schur ? XB + e * xp : XD[e];
          double* own = schur ? Xn + j * xp + e : X + j * xp + LB + e;
          init = *own;
          dst = all ? &S[e][t] : own;
        }
        double s = 0.0;
        for (int l = t8; l < terms; l += ks) s = fma(a[l], b[l], s);
        for (int o = 1; o < ks; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (live) {
          const double v = init - s;
          if (all) {
            for (int w = t8; w < nc; w += ks) st_cluster(cluster_addr(dst, w), v);
          } else if (t8 == 0) {
            *dst = v;
          }
        }
      }
      __syncwarp();
      cluster_sync();                                // the next leaf is in S, the rows are up to date
    }
  }
  pdl_trigger();
}

template <int G, int NT>
void launch_rows_g(double* X, int rows, const double* P, long long lda, int w, const double* ws,
                   cudaStream_t s) {
  const dim3 grid((rows + NT / G - 1) / (NT / G)), block(NT);
  switch ((w + LB - 1) / LB) {
    case 1: launch_k(panel_rows_kernel<G, 1, NT>, grid, block, 0, s, X, rows, P, lda, w, ws); break;
    case 2: launch_k(panel_rows_kernel<G, 2, NT>, grid, block, 0, s, X, rows, P, lda, w, ws); break;
    case 3: launch_k(panel_rows_kernel<G, 3, NT>, grid, block, 0, s, X, rows, P, lda, w, ws); break;
    case 4: launch_k(panel_rows_kernel<G, 4, NT>, grid, block, 0, s, X, rows, P, lda, w, ws); break;
    default: launch_k(panel_rows_kernel<G, 5, NT>, grid, block, 0, s, X, rows, P, lda, w, ws); break;
  }
}

}  // namespace

namespace {
}  // namespace

bool panel_wide_clusters() {
  static const bool ok = widest_cluster(panel_tile_kernel<15, PANEL_TILE>, 0, TILE_THREADS) == 16;
  return ok;
}

// One CTA for a single leaf; else a cluster of 16, or of 8 where the device
// has too few places for 16.
void launch_panel_tile(double* P, long long lda, int w, double* ws, int col0, DevStatus* st,
                       cudaStream_t s, int wait_polls, bool narrow) {
  if (w <= 0) return;
  const int polls = wait_polls > 0 ? wait_polls : LEAF_WAIT_POLLS;
  const bool wide = w > LB && !narrow && panel_wide_clusters();
  const dim3 n(w <= LB ? 1 : wide ? 16 : 8);
  auto* kern = w <= PANEL_TILE - PANEL_LEAF
                   ? (wide ? panel_tile_kernel<15, PANEL_TILE - PANEL_LEAF>
                           : panel_tile_kernel<7, PANEL_TILE - PANEL_LEAF>)
                   : (wide ? panel_tile_kernel<15, PANEL_TILE> : panel_tile_kernel<7, PANEL_TILE>);
  if (wide) allow_wide_clusters(kern, 0);  // an attribute of the current device
  launch_k_cluster(kern, n, dim3(TILE_THREADS), n, 0, s, P, lda, w, ws, col0, st, polls);
}

// G lanes a row and four or eight warps: 4 / 8 / 16 rows a CTA, the fewest that
// still let the SMs take all rows at once (a CTA's time grows with its rows;
// two CTAs on an SM share its FP64 units).  16 rows go as two warps a
// sub-partition of two rows each: 6% more instructions than one warp of four, but
// one warp's shuffles and shared-memory reads run behind the other's FMAs
// (1872 rows of 128 columns: 67 -> 48 us; the FMAs alone, spread evenly, 32).
void launch_panel_rows(double* X, int rows, const double* P, long long lda, int w,
                       const double* ws, cudaStream_t s) {
  if (rows <= 0 || w <= 0) return;
  if (rows <= 4 * GB300_SMS) launch_rows_g<32, 128>(X, rows, P, lda, w, ws, s);
  else if (rows <= 8 * GB300_SMS) launch_rows_g<16, 128>(X, rows, P, lda, w, ws, s);
  else launch_rows_g<16, 256>(X, rows, P, lda, w, ws, s);
}

// One CTA does blocks of up to 12 rows as fast as eight; sixteen beat eight from ~32
// columns (42: 19 against 20 us a block, 64: 29 against 35).  The line at 64 is the
// kernel's two leaves; there it is still ahead of the separate launches (37 us).
int chain_factor_ctas(const BtaShape& sh) {
  if (sh.ns > CHAIN_MAX_NS || sh.ns + sh.nd > CHAIN_MAX_ROWS) return 0;
  static const int widest = widest_cluster(chain_factor_kernel, CHAIN_FACTOR_SMEM, CHAIN_THREADS);
  if (!widest) return 0;
  return sh.ns + sh.nd <= 12 ? 1 : sh.ns + sh.nd <= 28 ? 8 : widest;
}

void launch_chain_factor(const BtaShape& sh, int nc, double* MF, DevStatus* st, cudaStream_t s,
                         int wait_polls) {
  const ChainShape z((int)sh.ns, (int)sh.nd, nc);
  allow_wide_clusters(chain_factor_kernel, CHAIN_FACTOR_SMEM);  // an attribute of the current device
  launch_k_cluster(chain_factor_kernel, dim3(nc), dim3(CHAIN_THREADS), dim3(nc),
                   z.elems((int)sh.ns, nc) * sizeof(double), s, MF, (int)sh.ns, (int)sh.nd, sh.nt, st,
                   wait_polls > 0 ? wait_polls : LEAF_WAIT_POLLS);
}

}  // namespace rgf
