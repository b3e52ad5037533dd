// Device helpers shared by the kernels of librgf_gb300 (include from .cu only).
#pragma once

#include <cstdint>

namespace rgf {

// ---- thread-block clusters and shared-memory hand-offs ------------------------
// Every thread of the cluster arrives and waits; shared-memory writes before
// it are visible to the cluster's reads after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
// *p of the cluster's CTA `rank` (p: this CTA's shared memory)
__device__ __forceinline__ double ld_cluster(const double* p, int rank) {
  unsigned a;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared-memory address of `p` (this CTA's) in the cluster's CTA `rank`
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ long long ld_cluster_i64(unsigned addr) {
  long long v;
  asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// ---- asynchronous copies of doubles from global to this CTA's shared memory ------
__device__ __forceinline__ void cp_async8(void* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
               :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// ---- FP64 arithmetic off the FP64 units ----------------------------------------
// float -> double by bit manipulation (no FP64 conversion instruction);
// zero and subnormal floats give zero
__device__ __forceinline__ double f2d_bits(float f) {
  const unsigned int u = __float_as_uint(f);
  const unsigned int ex = (u >> 23) & 0xffu;
  if (ex == 0) return 0.0;
  return __longlong_as_double((long long)((unsigned long long)(u >> 31) << 63 |
                                          (unsigned long long)(ex - 127 + 1023) << 52 |
                                          (unsigned long long)(u & 0x7fffffu) << 29));
}

// Reciprocal square root of a normal positive double with few dependent FP64
// operations (they are the slow link of the leaf's pivot chain): d = m 4^k
// with m in [1, 4) by integer ops; an FP32 seed y0 = rsqrt(m_hi) is refined
// once in double-float arithmetic on the FP32 units (m = m_hi + m_lo split
// exactly from the bit pattern; e = 1 - m y0^2 with FMA-exact products), which
// gives ~44 bits; one FP64 Newton step then gives full precision.  FP64 ops on
// the chain: one add, one multiply, two FMAs; the 4^-k scale is an exponent
// shift.
__device__ __forceinline__ double rsqrt_fast(double d) {
  const long long b = __double_as_longlong(d);
  const int e = (int)((b >> 52) & 0x7ff) - 1023;
  if (e == -1023) return 1.0 / sqrt(d);                   // subnormal pivot
  const int k = e >> 1;                                   // d = m * 4^k, m in [1, 4)
  const long long mb = b - ((long long)(2 * k) << 52);
  const double m = __longlong_as_double(mb);
  const int em = (int)((mb >> 52) & 0x7ff) - 1023;        // 0 or 1
  // m_hi: the top 24 significant bits as a float; m_lo: the remaining 29 bits
  const float mh = __uint_as_float((unsigned int)(((mb >> 52) - 1023 + 127) << 23) |
                                   (unsigned int)((mb >> 29) & 0x7fffff));
  const float ml = (float)(unsigned int)(mb & ((1ll << 29) - 1)) *
                   __uint_as_float((unsigned int)(127 + em - 52) << 23);
  const float y0 = rsqrtf(mh);
  const float p = y0 * y0;
  const float pe = fmaf(y0, y0, -p);                      // y0^2 = p + pe exactly
  float t = fmaf(-mh, p, 1.0f);
  t = fmaf(-mh, pe, t);
  t = fmaf(-ml, p, t);                                    // e = 1 - m y0^2
  const double y1 = f2d_bits(y0) + f2d_bits(0.5f * y0 * t);
  const double hm = __longlong_as_double(mb - (1ll << 52));  // m / 2, exact
  const double y2 = fma(y1, fma(-hm, y1 * y1, 0.5), y1);    // y1 (1.5 - m y1^2 / 2)
  return __longlong_as_double(__double_as_longlong(y2) - ((long long)k << 52));
}

}  // namespace rgf
