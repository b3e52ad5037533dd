// Internal interfaces shared by the CUDA translation units of librgf_gb300.
#pragma once

#include <vector>

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace rgf {

// Lives in device memory, one per handle.  Kernels record failures here
// instead of trapping; the host reads it after each stage.
struct DevStatus {
  int not_spd_col;   // smallest global column with a non-positive pivot (INT32_MAX: none)
  int bad_input;     // ingest saw an entry outside the block pattern
  int timeout;       // a bounded device-side wait gave up
  int pad;
};

// What the host reads after a stage, in one copy.
struct DevResults {
  DevStatus status;
  double scalars[8];  // [0] logdet, [1] ||r||, [2] ||b||
};

constexpr int GB300_SMS = 152;  // the splits of FP64 work over the chip are fitted to it

// ---- programmatic dependent launch -------------------------------------------
// Kernels are launched with programmatic stream serialization (launch_k): the
// next kernel in a stream may be scheduled once every CTA of the running one
// has called pdl_trigger() (placed after each kernel's main loop, so the next
// kernel's CTAs become resident during the tail instead of after it), and
// every kernel calls pdl_wait() before its first global memory access, which
// returns once the previous kernel in the stream has completed and its writes
// are visible.  Both are no-ops in a kernel launched without the attribute.
// RGF_GB300_PDL=0 launches without it.
// Launches inside a NoPdl scope of this thread go without it too: those of the
// look-ahead side stream (their early CTAs would wait on SMs that the main
// stream's kernels need), and, while that stream has work, the diagonal tiles
// and FP64 products of the main one (a tile that comes in early sits on an SM
// whose FP64 units another product is still using).  Factorization replayed as
// a graph with / without those attributes: ns = 2000, nt = 10 split 32.1 / 28.8 ms,
// ns = 515, nt = 20 split 10.7 / 9.1 ms, ns = 333, nt = 20 FP64 7.9 / 7.2 ms.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

bool pdl_enabled();
bool& pdl_scope();  // this thread launches with the attribute (default true)
struct NoPdl {
  bool before;
  explicit NoPdl(bool off) : before(pdl_scope()) { pdl_scope() = before && !off; }
  ~NoPdl() { pdl_scope() = before; }
};

// launch_k_cluster: the same with thread-block clusters of the given size.
template <typename... KArgs, typename... Args>
inline void launch_k_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, dim3 cluster,
                             size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  cfg.attrs = at;
  cfg.numAttrs = 0;
  if (cluster.x * cluster.y * cluster.z > 1) {
    at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    at[cfg.numAttrs].val.clusterDim.x = cluster.x;
    at[cfg.numAttrs].val.clusterDim.y = cluster.y;
    at[cfg.numAttrs].val.clusterDim.z = cluster.z;
    cfg.numAttrs++;
  }
  // created streams only: not the default streams (the legacy one synchronizes
  // with every stream)
  if (pdl_enabled() && pdl_scope() && s != nullptr && s != cudaStreamLegacy && s != cudaStreamPerThread) {
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs++;
  }
  cudaLaunchKernelEx(&cfg, kern, args...);  // a failure stays the pending launch error
}

template <typename... KArgs, typename... Args>
inline void launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                     Args... args) {
  launch_k_cluster(kern, grid, block, dim3(1, 1, 1), smem, s, args...);
}

// `bytes` of shared memory and clusters of 16 for the kernel on the current device
template <typename K>
bool allow_wide_clusters(K* kern, size_t bytes) {
  if (!cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) &&
      !cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))
    return true;
  cudaGetLastError();
  return false;
}
// How many CTAs of the kernel a cluster can have with `bytes` of shared memory each: 16
// (more than the portable size), else 8, or 0.
template <typename K>
int widest_cluster(K* kern, size_t bytes, int threads) {
  if (!allow_wide_clusters(kern, bytes)) return 0;
  for (int nc = 16; nc >= 8; nc /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bytes;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) cudaGetLastError();
    else if (n >= 4) return nc;  // not only a corner of the chip
  }
  return 0;
}

enum Tri { TRI_NONE = 0, TRI_LOWER = 1, TRI_UPPER = 2 };

// D = alpha * op(A) * op(B) + beta * C, column-major, op(A) m x k, op(B) k x n.
// triA/triB declare a triangular operand (of op(X)); its other triangle is
// treated as zero whatever memory holds.  outLower writes only r >= c; output
// tiles with nothing to write are not computed.
// batch > 1 runs independent problems offset by sA/sB/sC/sD elements.
struct GemmDesc {
  int m = 0, n = 0, k = 0;
  const double* A = nullptr; long long lda = 0; int transA = 0;
  // Rows >= mA1 of A come from A2 (row r at A2 + (r - mA1), same lda and
  // batch stride): a stacked operand whose two row blocks are not adjacent
  // in memory.  transA == 0 only; A2 == nullptr means one block.
  const double* A2 = nullptr; int mA1 = 0;
  // Rows >= mD1 of C and D live at C2 / D2 (row r at D2 + (r - mD1), same
  // leading dimensions and batch strides); D2 == nullptr means one block.
  const double* C2 = nullptr; double* D2 = nullptr; int mD1 = 0;
  const double* B = nullptr; long long ldb = 0; int transB = 0;
  const double* C = nullptr; long long ldc = 0;
  double* D = nullptr; long long ldd = 0;
  double alpha = 1.0, beta = 0.0;
  int triA = TRI_NONE, triB = TRI_NONE, outLower = 0;
  int batch = 1;
  long long sA = 0, sB = 0, sC = 0, sD = 0;
  int ksplit = 1;       // FP64 kernel: set by the launcher
  bool beside = false;  // FP64 kernel: other work shares the GPU
  bool early = false;   // FP64 kernel: the stream's previous kernel does not write A (a
                        // product of the block substitution)
  int tile = 0;  // FP64 kernel: output tile 32 or 64; 0 = chosen by the launcher
};

// Whether the t x t output tile at (m0, n0) has anything to write.
inline bool tile_written(int outLower, int m0, int n0, int t) { return !(outLower && m0 + t <= n0); }
// The i-th of the written tiles, column by column (nx tiles to a full column).
struct TilePos {
  int x, y;
};
__device__ inline TilePos tile_at(int outLower, int nx, int i) {
  if (!outLower) return {i % nx, i / nx};
  int y = 0;
  while (i >= nx - y) i -= nx - y++;
  return {i + y, y};
}
// Number of t x t tiles of the m x n output that are written (one batch item).
inline long long tiles_written(const GemmDesc& g, int t) {
  long long tiles = 0;
  for (int m0 = 0; m0 < g.m; m0 += t)
    for (int n0 = 0; n0 < g.n; n0 += t) tiles += tile_written(g.outLower, m0, n0, t);
  return tiles;
}

// Algorithmic flops of one GemmDesc (triangular operands and lower-only
// outputs counted at their LAPACK sizes).
double gemm_flops(const GemmDesc& g);

// ---- complex Hermitian matrices (hermitian.cu) -------------------------------
// Lower CSC of the real symmetric embedding [[X, -Y], [Y, X]] of the Hermitian
// A = X + iY given as its lower CSC (a: interleaved re, im), ordered so that it
// is a BTA matrix with (2ns, nt, 2nd).
int hermitian_embed(const size_t* ia, const size_t* ja, const double* a, size_t ns, size_t nt,
                    size_t nd, std::vector<size_t>& ia2, std::vector<size_t>& ja2,
                    std::vector<double>& a2);
// Real index of Re (imag = 0) or Im (imag = 1) of complex unknown k.
size_t hermitian_real_index(size_t ns, size_t nt, size_t nd, size_t k, int imag);

// ---- FP64 kernels (k_fp64.cu) ---------------------------------------------
// Returns the number of kernels launched.
int launch_gemm_fp64(const GemmDesc& g, cudaStream_t s);

// ---- panel factorization (k_panel.cu) -------------------------------------------
// Cholesky of the w x w (w <= PANEL_TILE) lower tile at P (column-major, lda), in
// place.  Records the first non-positive pivot (global column col0 + j) in st.
// Each wait of a column for the previous pivot polls at most wait_polls times
// (0 = LEAF_WAIT_POLLS); a wait that runs out records a timeout in st and the
// tile's leaves stop updating.  ws (PANEL_WS doubles) receives what
// launch_panel_rows reads: per 32-column leaf its unit columns, then d^{-1/2}.
constexpr int PANEL_LEAF = 32, PANEL_TILE = 160;
constexpr int PANEL_LEAF_WS = PANEL_LEAF * PANEL_LEAF + PANEL_LEAF;
constexpr int PANEL_WS = PANEL_TILE / PANEL_LEAF * PANEL_LEAF_WS;
constexpr int LEAF_WAIT_POLLS = 1 << 26;
// narrow: a cluster of 8 CTAs even where the device has room for 16.
void launch_panel_tile(double* P, long long lda, int w, double* ws, int col0, DevStatus* st,
                       cudaStream_t s, int wait_polls = 0, bool narrow = false);
// Whether clusters of 16 CTAs of that launch can be resident on this device.
bool panel_wide_clusters();
// X := X L^{-T} for `rows` rows of w columns at X (leading dimension lda), L the
// tile factored by launch_panel_tile at P (same lda) with its ws.
void launch_panel_rows(double* X, int rows, const double* P, long long lda, int w,
                       const double* ws, cudaStream_t s);

// ---- chains of small blocks (k_chain.cu) -----------------------------------------
struct BtaShape {
  long long ns, nt, nd, n;
};
// Factorization of all block columns (not the corner) in one launch, for
// ns <= CHAIN_MAX_NS and ns + nd <= CHAIN_MAX_ROWS (k_panel.cu); MF holds A on entry.
// Status and waits as launch_panel_tile.
constexpr int CHAIN_MAX_NS = 64, CHAIN_MAX_ROWS = 72;
// CTAs of that launch's cluster, 0 where the blocks are too large for it.
int chain_factor_ctas(const BtaShape& sh);
void launch_chain_factor(const BtaShape& sh, int nc, double* MF, DevStatus* st, cudaStream_t s,
                         int wait_polls = 0);
// Selected inversion of all blocks in one launch, for ns + nd <= SELINV_CHAIN_MAX: on
// entry MS holds Q_i = U_i U_i^T (lower) in its diagonal blocks and Sigma_dd in the corner;
// K the K_i of blocks 0 .. nt-2, Klast that of the last one (nd x ns).
constexpr int SELINV_CHAIN_MAX = 72;
constexpr int SELINV_CHAIN_SMEM = 180 * 1024, CHAIN_FACTOR_SMEM = 64 * 1024;  // at most
// CTAs of that launch's cluster, 0 where the blocks are too large for it.
int selinv_chain_ctas(const BtaShape& sh);
void launch_selinv_chain(const BtaShape& sh, int nc, const double* K, const double* Klast,
                         double* MS, cudaStream_t s);

// The block substitution of nrhs right-hand sides in one launch: R holds b on entry and x
// on return, Y is scratch (both n x nrhs); U the inverses of all diagonal blocks and of
// the corner.
constexpr int SOLVE_CHAIN_MAX = 320, SOLVE_CHAIN_SMEM = 200 * 1024;
// CTAs of that launch's cluster, 0 where separate products are the better way.
int solve_chain_ctas(const BtaShape& sh, int nrhs);
void launch_solve_chain(const BtaShape& sh, int nc, const double* MF, const double* U, double* R,
                        double* Y, int nrhs, cudaStream_t s);

// Every device allocation of the library goes through here (so that a test
// can make one fail: rgf_debug_fail_alloc_after).  cudaMalloc semantics.
// On a thread that has a device arena set (set_thread_arena), memory comes
// from the arena instead, with no cudaMalloc (and device_free returns it
// there, with no cudaFree and its device-wide wait).
cudaError_t device_malloc(void** p, size_t bytes);
void device_free(void* p);

// A device arena: one cudaMalloc of `bytes` at creation, then first-fit
// sub-allocation (256-byte aligned, neighbours merged on free) under a mutex.
// When it cannot serve a request (full or fragmented) device_malloc falls back
// to cudaMalloc and counts it.
struct DeviceArena;
DeviceArena* arena_create(size_t bytes, int* status);
void arena_destroy(DeviceArena* a);
void set_thread_arena(DeviceArena* a);
long long arena_fallbacks(DeviceArena* a);
size_t arena_in_use(DeviceArena* a);

// Row-parallel triangular solve with an nbk x nbk (nbk <= 64) lower tile L:
//   mode 0: X := X * L^{-T}   (forward,  "R L T N")
//   mode 1: X := X * L^{-1}   (backward, "R L N N")
// X has `rows` independent rows; element (r, j) at X[r*xrs + j*xcs].
// batch > 1: problem b uses X + b*sX, L + b*sL.
void launch_trsm_rows(double* X, long long xrs, long long xcs, int rows, const double* L,
                      long long ldl, int nbk, int mode, int batch, long long sX, long long sL,
                      cudaStream_t s);

// U = L^{-T} of every 64 x 64 diagonal tile (the last may be smaller) of the n x n
// lower factor L, for `batch` of them; only those tiles of U are written.
void launch_leaf_inverses(double* U, long long ldu, int n, const double* L, long long ldl,
                          int batch, long long sU, long long sL, cudaStream_t s);

// Measured FP64 (DMMA) throughput of the current device in TFLOP/s.
int measure_fp64_peak(double* tflops);

// ---- small kernels (k_misc.cu) ------------------------------------------------
long long mf_col_offset(const BtaShape& sh, long long i);
long long mf_lda(const BtaShape& sh, long long i);
long long mf_dense_row(const BtaShape& sh, long long i);
// Blocks whose K_i = [L_{i+1,i}; C_i] L_ii^{-1} the selected inversion forms in one
// batch: as many as fit K_CHUNK_BYTES (four blocks of ns = 2000), at least one.
constexpr size_t K_CHUNK_BYTES = (size_t)128 << 20;
long long selinv_chunk(const BtaShape& sh);

// Scatter the device CSC into the (pre-zeroed) MF layout; one warp per column.
// Columns [c_lo, c_hi) only (c_hi < 0: to the last column): every entry of a
// column lands in its own block column's panel.
void launch_ingest(const BtaShape& sh, const size_t* ia, const size_t* ja, const double* a,
                   double* MF, DevStatus* st, cudaStream_t s, long long c_lo = 0,
                   long long c_hi = -1);
// Sum of nparts partial log sums, times 2, in a fixed order -> *out.
// *out = 2 sum(log diag(L)) over the factor MF: per-block sums into parts
// (logdet_parts(sh) of them), then a fixed-order total.
int logdet_parts(const BtaShape& sh);
void launch_logdet(const BtaShape& sh, const double* MF, double* parts, double* out,
                   cudaStream_t s);
// diag[k] = MS[diag position of k] for all k < n.
void launch_extract_diag(const BtaShape& sh, const double* MS, double* diag, cudaStream_t s);
// batch of identity matrices (m x m, ld) at X + b*stride
void launch_set_identity(double* X, long long ld, int m, int batch, long long stride,
                         cudaStream_t s);
// Upper triangle of the symmetric n x n matrix X from its lower triangle; with S
// (may be null) also the full symmetric
// [X, Xd^T; Xd, Sdd] into S ((n + nd) x (n + nd), packed), Xd (nd x n, ld) its
// arrowhead rows and Sdd nd x nd.
void launch_mirror_sigma(double* X, long long ld, int n, const double* Xd, const double* Sdd,
                         int nd, double* S, cudaStream_t s);
// r = b - A x (symmetric, from the lower CSC) for the first column; then
// out[0] = ||r||_2, out[1] = ||b||_2 (scaled sums of squares, as dnrm2).
// scratch: n doubles.  CSC entries outside the lower triangle or past row n-1
// are skipped; with `bad` (device int, may be null) they set *bad and both
// outputs become NaN.  Returns the first launch error (the caller's pending
// errors are the caller's to check first).
cudaError_t launch_residual(long long n, const size_t* ia, const size_t* ja, const double* a,
                            const double* x, const double* b, double* scratch, double* out,
                            int* bad, cudaStream_t s);
// R = B - A X for nrhs columns (ld n) from the lower CSC; Y is n*nrhs scratch
void launch_residual_vectors(long long n, int nrhs, const size_t* ia, const size_t* ja,
                             const double* a, const double* X, const double* B, double* Y,
                             double* R, cudaStream_t s);
// out[2q] = ||R[:, q]||_2, out[2q + 1] = ||B[:, q]||_2 (columns n apart,
// scaled sums of squares) for q < nrhs.
void launch_rhs_norms(long long n, int nrhs, const double* R, const double* B, double* out,
                      cudaStream_t s);
// right-hand sides per pass of the multi-RHS SpMV of launch_residual_vectors
constexpr int SPMV_MAX_RHS = 16;
// x += d over len entries
void launch_add(long long len, double* x, const double* d, cudaStream_t s);
// corner -= sum_i C_i C_i^T (lower part) over all block columns, for
// 0 < nd <= ARROW_SYRK_MAX_ND: partial sums over 256 columns of block columns
// into partial (arrow_syrk_elems doubles), then added in a fixed order.
constexpr int ARROW_SYRK_MAX_ND = 32;
long long arrow_syrk_elems(const BtaShape& sh);
void launch_arrow_syrk(const BtaShape& sh, double* MF, double* partial, cudaStream_t s);
// out[q*ldo + dd] = sum_i sum_j C_i(dd, j) * R_i(j, q) over block columns,
// computed as per-block partials then an ordered sum: the arrowhead part of
// the forward solve.  y_d -= that.
void launch_arrow_gemv(const BtaShape& sh, const double* MF, const double* rhs, long long ldr,
                       int nrhs, double* partial, cudaStream_t s);
void launch_arrow_reduce(const BtaShape& sh, const double* partial, int nrhs, double* rhs,
                         long long ldr, cudaStream_t s);

}  // namespace rgf
