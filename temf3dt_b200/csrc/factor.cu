// K2 + K3: step-matrix formation and supernodal numeric Cholesky on the GPU.
//
// Replaces mkl_add_3 + mkl_to_csr (src/FETD_FWD.f90:2006-2039, 1974-2004)
// and the numeric part of PARDISO phase 12 (src/FETD_UTILITY.f90:912-917,
// mtype 2 = real SPD).  A(dt) = 0*A_eps + 3*M_sigma + 2*dt*K is formed
// directly into the supernodal panels (the pattern is dt-independent).
//
// Schedule: bottom-up levels of the supernodal elimination tree.  Per level:
//   k_potrf      : one CTA per supernode: dense Cholesky of the (<=64 x 64)
//                  diagonal block, 8 columns at a time;
//   k_trsm       : the below-diagonal rows solved against it, 64 rows per
//                  CTA, 16 columns at a time;
//   k_update     : the Schur update L21 L21^T of every supernode of the level,
//                  in tiles of 64x64 or 32x32 on the FP64 tensor cores (DMMA
//                  mma.sync.m8n8k4.f64), scattered into the ancestor panels
//                  through precomputed relative indices with FP64 atomics
//                  (red.global.add.f64), on every level: launches overlap.
// Supernodes of one level may update the same ancestor entry, in the order in
// which their tiles finish: the last bit of such an entry differs from run to
// run, and through the air's 1e-12 S/m so do the edge vectors, by 1e-9 to 1e-8
// of their norm.  A level without such entries runs its updates in two launches
// on two streams, behind the next level's blocks (launch_factor_values).
// Pivot failures are reported through a status word (first failing column),
// never by trapping.
#include <algorithm>
#include <climits>

#include "dmma.cuh"
#include "factor.h"

namespace temf {

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__global__ void k_load_A(int64_t n, const int* __restrict__ src, const int64_t* __restrict__ dst,
                         const double* __restrict__ M, double a, const double* __restrict__ K, double b,
                         double* __restrict__ L) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int p = src[q];
  L[dst[q]] = a * M[p] + (K ? b * K[p] : 0.0);
}

// Dense Cholesky of the (<= 64 x 64) diagonal block of each supernode of a level.
//
// sgn != null: the indefinite mode, A = L S L^T with S = diag(+-1) (sgn, in
// the permuted order) and L_kk = sqrt(|d_k|) > 0, the sign of the pivot d_k in
// s_k.  A pivot that cancels below kPivotTol of its column's diagonal entry
// as the block's elimination starts (or is not finite) is perturbed to that
// size (static pivot perturbation, counted in status[2]); the iterative
// refinement of the solves recovers the accuracy.  The first non-positive
// pivot is recorded in status[0] in both modes.
constexpr double kPivotTol = 1e-13;

constexpr int kPotrfThreads = 256;  // warps 0-1: the panel's rows; the others: the columns after it, finished columns out
constexpr int kPanel = 8;           // columns eliminated between two trailing updates
constexpr int kLdD = kSnCols + 2;   // row stride of the block in shared memory: column reads and DMMA fragments 2-way

struct PotrfShared {
  double D[kSnCols][kLdD];
  double diag[kSnCols];  // L_kk
  double dinv[kSnCols];  // 1 / L_kk
  double sg[kSnCols];    // sign of the pivot (1 unless indefinite)
  double d0[kSnCols];    // diagonal entries as the block's elimination starts
};

// Panel p, 8 columns, by warps 0 and 1: lane l of warp w owns row 32 w + l.
//  1. The panel's entries get the rank-8 update of the panel before (earlier
//     ones are in already), in registers.
//  2. Every lane eliminates the panel's 8 x 8 diagonal block redundantly, so
//     the chain per column is the square root, its reciprocal, a multiply and
//     an FMA, with nothing to broadcast (a 64-bit shuffle issues in 11 cycles
//     on sm_100a, a warp's FP64 FMA in 3).
//  3. Each lane substitutes its own row.
// Every entry gets the FMAs of column-by-column elimination in ascending
// column order: the same rounding whatever the panel width.
template <bool kIndef>
__device__ __forceinline__ void potrf_panel(PotrfShared& S, int p, int c, int f, int* status, double* sgn) {
  const int row = threadIdx.x, j0 = kPanel * p;  // threadIdx.x < 64
  double a[kPanel];
#pragma unroll
  for (int k = 0; k < kPanel; ++k) a[k] = S.D[row][j0 + k];
  if (p > 0) {
    const int i0 = j0 - kPanel;
    double l[kPanel];
#pragma unroll
    for (int k = 0; k < kPanel; ++k) l[k] = kIndef ? S.D[row][i0 + k] * S.sg[i0 + k] : S.D[row][i0 + k];
#pragma unroll
    for (int j = 0; j < kPanel; ++j)
#pragma unroll
      for (int k = 0; k < kPanel; ++k) a[j] -= l[k] * S.D[j0 + j][i0 + k];
#pragma unroll
    for (int k = 0; k < kPanel; ++k)
      if (row >= j0 && row < j0 + kPanel) S.D[row][j0 + k] = a[k];
  }
  asm volatile("bar.sync 1, 64;\n" ::: "memory");
  double t[kPanel][kPanel], inv[kPanel], sg[kPanel], mydiag = 0.0, myinv = 0.0, mysg = 1.0;
#pragma unroll
  for (int i = 0; i < kPanel; ++i)
#pragma unroll
    for (int k = 0; k <= i; ++k) t[i][k] = S.D[j0 + i][j0 + k];
  int bad = INT_MAX, npert = 0;
#pragma unroll
  for (int k = 0; k < kPanel; ++k) {
    double d = t[k][k];
    sg[k] = 1.0;
    if (!(d > 0.0) && j0 + k < c) bad = min(bad, j0 + k);  // non-positive or NaN pivot
    if (kIndef) {
      sg[k] = d < 0.0 ? -1.0 : 1.0;
      d = fabs(d);
      const double d0 = S.d0[j0 + k];
      const double tau = kPivotTol * (d0 > 0.0 ? d0 : 1.0);
      if (!(d >= tau) || !(d <= 1e300)) {  // cancelled, NaN or infinite pivot: perturb
        d = tau;
        npert += j0 + k < c ? 1 : 0;
      }
    } else {
      d = d > 0.0 ? d : 1.0;  // continue with 1; the factor is reported invalid
    }
    const double lkk = sqrt(d);
    inv[k] = 1.0 / lkk;
    if (row == j0 + k) {
      mydiag = lkk;
      myinv = inv[k];
      mysg = sg[k];
    }
    if (kIndef) inv[k] *= sg[k];
#pragma unroll
    for (int i = k + 1; i < kPanel; ++i) t[i][k] *= inv[k];
#pragma unroll
    for (int j = k + 1; j < kPanel; ++j)
#pragma unroll
      for (int i = j; i < kPanel; ++i) t[i][j] -= (kIndef ? t[i][k] * sg[k] : t[i][k]) * t[j][k];
  }
#pragma unroll
  for (int k = 0; k < kPanel; ++k) {
    a[k] *= inv[k];
#pragma unroll
    for (int j = k + 1; j < kPanel; ++j) a[j] -= (kIndef ? a[k] * sg[k] : a[k]) * t[j][k];
  }
  asm volatile("bar.sync 1, 64;\n" ::: "memory");  // the diagonal block has been read
#pragma unroll
  for (int k = 0; k < kPanel; ++k)
    if (row > j0 + k) S.D[row][j0 + k] = a[k];
  if (row >= j0 && row < j0 + kPanel) {
    S.diag[row] = mydiag;
    S.dinv[row] = myinv;
    S.sg[row] = mysg;
    if (kIndef && row < c) sgn[f + row] = mysg;
  }
  if (row == 0) {
    if (bad != INT_MAX) atomicMin(status, f + bad + 1);
    if (kIndef && npert) atomicAdd(status + 2, npert);
  }
}

// Tile (I, J) of 8 x 8 minus the products with panel p.  The tile is the
// accumulator: a DMMA adds its four products one FMA after the other in
// ascending k, as column-by-column elimination does.
__device__ __forceinline__ void potrf_tile(PotrfShared& S, int I, int J, int p) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int ri = 8 * I + g, rj = 8 * J;
  double x0 = S.D[ri][rj + 2 * q], x1 = S.D[ri][rj + 2 * q + 1];
#pragma unroll
  for (int k0 = 0; k0 < kPanel; k0 += 4) {
    const int k = kPanel * p + k0 + q;
    dmma_8x8x4(x0, x1, -S.D[ri][k] * S.sg[k], S.D[rj + g][k]);
  }
  S.D[ri][rj + 2 * q] = x0;
  S.D[ri][rj + 2 * q + 1] = x1;
}

// One CTA per block, bound by the 64-step pivot chain.  While warps 0 and 1
// eliminate panel p, the others apply panel p - 1 to the columns after p
// (DMMA) and write the finished columns of panel p - 1: the panel's block, and
// the sweeps' copy (row i scaled by 1/L_ii, 1/L_ii on the diagonal, zeros
// above; c x c, column-major).  A 64 x 64 block in its stream takes 14.4 us;
// column by column with two barriers, a square root and a division per
// column it took 73.  Two CTAs per SM: the bottom levels hold hundreds of
// narrow blocks.
template <bool kIndef>
__global__ void __launch_bounds__(kPotrfThreads, 2) k_potrf(
    const int* __restrict__ level_sn, const int* __restrict__ sn_first,
    const int64_t* __restrict__ rows_ptr, const int64_t* __restrict__ Lptr, double* __restrict__ L,
    int* __restrict__ status, double* __restrict__ sgn, const int64_t* __restrict__ Dptr) {
  __shared__ PotrfShared S;
  const int s = level_sn[blockIdx.x];
  const int f = sn_first[s];
  const int c = sn_first[s + 1] - f;
  const int64_t r = rows_ptr[s + 1] - rows_ptr[s];
  const int64_t ld = c + r;
  double* P = L + Lptr[s];
  double* Q = L + Dptr[s];
  const int tid = threadIdx.x, i = tid & (kSnCols - 1);
  const int np = (c + kPanel - 1) / kPanel;
  // lower triangle; zeros above it and past c
#pragma unroll 16
  for (int j = tid / kSnCols; j < np * kPanel; j += kPotrfThreads / kSnCols)
    S.D[i][j] = (i < c && j <= i) ? P[(int64_t)j * ld + i] : 0.0;
  if (tid < kSnCols) S.sg[tid] = 1.0;
  __syncthreads();
  if (kIndef) {
    if (tid < c) S.d0[tid] = fabs(S.D[tid][tid]);
    __syncthreads();
  }
  // columns of panel p out, by `nt` threads from `t0` on
  auto out = [&](int p, int t0, int nt) {
    if (i >= c) return;
    for (int j = kPanel * p + (tid - t0) / kSnCols; j < min(c, kPanel * (p + 1)); j += nt / kSnCols)
      if (i >= j) P[(int64_t)j * ld + i] = i > j ? S.D[i][j] : S.diag[i];
  };
  for (int p = 0; p <= np; ++p) {
    if (tid < 64) {
      if (p < np) potrf_panel<kIndef>(S, p, c, f, status, sgn);
    } else if (p > 0) {
      int t = (tid >> 5) - 2;
      for (int J = p + 1; J < np; ++J)
        for (int I = J; I < np; ++I, ++t)
          if (t % 6 == 0) potrf_tile(S, I, J, p - 1);
      out(p - 1, 64, kPotrfThreads - 64);
    }
    __syncthreads();
  }
  if (i < c) {
    const double di = S.dinv[i];
    for (int j = tid / kSnCols; j < c; j += kPotrfThreads / kSnCols)
      Q[(int64_t)j * c + i] = i > j ? S.D[i][j] * di : (i == j ? di : 0.0);
  }
}

// a / b correctly rounded, from y = 1 / b correctly rounded: two residual
// corrections of a y, the last of which rounds correctly (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990, theorem on quotients) while neither
// over- nor underflows: b one that divisor_fits() takes, the result finite and
// its quotient_key() at least kQuotientKey (a - q b is a double then).  The
// caller divides otherwise.  45 cycles on the chain of a row, a division 110.
__device__ __forceinline__ double quotient(double a, double b, double y) {
  double q = a * y;
  q = fma(-fma(q, b, -a), y, q);  // (in this form a zero keeps its sign)
  return fma(-fma(q, b, -a), y, q);
}
// square roots of positive doubles; not the infinite one, not NaN
__device__ __forceinline__ bool divisor_fits(double b) { return b >= 0x1p-537 && b <= 0x1p512; }
// grows with |q|, zeros on top: kQuotientKey for 2^-400
__device__ __forceinline__ unsigned quotient_key(double q) {
  return ((unsigned)__double2hiint(q) & 0x7fffffffu) - 1u + min((unsigned)__double2loint(q), 1u);
}
constexpr unsigned kQuotientKey = ((1023u - 400u) << 20) - 1u;

// Below-diagonal rows of the level's supernodes, kTrsmRows rows per CTA:
// x L11^T = a, L21 = x S11 in the indefinite mode (sgn != null).  Panels of 16
// columns: the products with the columns before a panel are DMMA tiles that
// start from the panel's entries (each entry gets its FMAs in ascending
// column order, as in a row-by-row substitution), then one thread per row
// substitutes inside the panel in registers.  A level of one 64-column block
// takes 13 us where one row per thread and a division per column took 36.
struct TrsmChunk {
  int s;
  int r0;
};
constexpr int kTrsmRows = 64;
constexpr int kTrsmThreads = 128;
constexpr int kTrsmPanel = 16;
constexpr int kLdX = kTrsmRows + 4;         // DMMA fragments (4 columns x 8 rows) without bank conflicts

inline size_t trsm_smem(int width) {        // X [w][kLdX], the block [w][kLdD], 1 / L_kk [w]; w: whole panels
  const int w = (width + kTrsmPanel - 1) / kTrsmPanel * kTrsmPanel;
  return (size_t)w * (kLdX + kLdD + 1) * sizeof(double);
}

// One row of a panel with divisions: infinities, NaN, values at the ends of the range.
__device__ __noinline__ void divide_panel(double* x, const double* D) {
  for (int j = 0; j < kTrsmPanel; ++j) {
    const double v = x[j * kLdX] / D[j * kLdD + j];
    x[j * kLdX] = v;
    for (int k = j + 1; k < kTrsmPanel; ++k) x[k * kLdX] -= v * D[k * kLdD + j];
  }
}

__global__ void __launch_bounds__(kTrsmThreads) k_trsm(const TrsmChunk* __restrict__ chunks,
                                                       const int* __restrict__ sn_first,
                                                       const int64_t* __restrict__ rows_ptr,
                                                       const int64_t* __restrict__ Lptr, double* __restrict__ L,
                                                       const double* __restrict__ sgn) {
  extern __shared__ __align__(16) double trsm_sm[];
  const TrsmChunk ch = chunks[blockIdx.x];
  const int s = ch.s;
  const int f = sn_first[s];
  const int c = sn_first[s + 1] - f;
  const int64_t r = rows_ptr[s + 1] - rows_ptr[s];
  const int64_t ld = c + r;
  double* P = L + Lptr[s];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int np = (c + kTrsmPanel - 1) / kTrsmPanel, w = np * kTrsmPanel;
  double* X = trsm_sm;              // [column][row]
  double* D = X + w * kLdX;         // [row of L11][column]; past c: zeros, ones on the diagonal
  double* rinv = D + w * kLdD;
  const int t = tid & (kTrsmRows - 1);
  const int64_t i = ch.r0 + t;
  const bool on = i < r;
  double* row = P + c + i;
#pragma unroll 8
  for (int j = tid / kTrsmRows; j < w; j += kTrsmThreads / kTrsmRows) {
    const double x = (on && j < c) ? row[(int64_t)j * ld] : 0.0;
    const double d = (t >= j && t < c) ? P[(int64_t)j * ld + t] : (t == j ? 1.0 : 0.0);
    X[j * kLdX + t] = x;
    if (t < w) D[t * kLdD + j] = d;
  }
  __syncthreads();
  if (tid < w) rinv[tid] = 1.0 / D[tid * kLdD + tid];
  const bool fits = __syncthreads_and(tid >= w || divisor_fits(D[tid * kLdD + tid]));
  for (int p = 0; p < np; ++p) {
    const int j0 = kTrsmPanel * p;
    if (p > 0) {  // rows 16 warp .. + 15 of the panel minus the products with the columns before it
      double acc[2][2][2];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) acc[a][b][e] = X[(j0 + 8 * b + 2 * q + e) * kLdX + 16 * warp + 8 * a + g];
#pragma unroll 4
      for (int k0 = 0; k0 < j0; k0 += 4) {
        double fa[2], fb[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) fa[a] = -X[(k0 + q) * kLdX + 16 * warp + 8 * a + g];
#pragma unroll
        for (int b = 0; b < 2; ++b) fb[b] = D[(j0 + 8 * b + g) * kLdD + k0 + q];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 2; ++b) dmma_8x8x4(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
      }
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) X[(j0 + 8 * b + 2 * q + e) * kLdX + 16 * warp + 8 * a + g] = acc[a][b][e];
      __syncthreads();
    }
    if (tid < kTrsmRows) {
      double x[kTrsmPanel];
#pragma unroll
      for (int j = 0; j < kTrsmPanel; ++j) x[j] = X[(j0 + j) * kLdX + t];
#pragma unroll
      for (int j = 0; j < kTrsmPanel; ++j) {
        x[j] = quotient(x[j], D[(j0 + j) * kLdD + j0 + j], rinv[j0 + j]);
#pragma unroll
        for (int k = j + 1; k < kTrsmPanel; ++k) x[k] -= x[j] * D[(j0 + k) * kLdD + j0 + j];
      }
      unsigned key = ~0u;
#pragma unroll
      for (int j = 0; j < kTrsmPanel; ++j) key = min(key, quotient_key(x[j]));
      // what is not finite has made the last column NaN
      if (!fits || key < kQuotientKey || !isfinite(x[kTrsmPanel - 1])) {
        divide_panel(X + j0 * kLdX + t, D + j0 * kLdD + j0);
#pragma unroll
        for (int j = 0; j < kTrsmPanel; ++j) x[j] = X[(j0 + j) * kLdX + t];
      }
#pragma unroll
      for (int j = 0; j < kTrsmPanel; ++j) {
        X[(j0 + j) * kLdX + t] = x[j];
        if (on && j0 + j < c) row[(int64_t)(j0 + j) * ld] = sgn ? x[j] * sgn[f + j0 + j] : x[j];
      }
    }
    __syncthreads();
  }
}

// The arithmetic that the factor's rounding rests on, one operand set per
// thread or warp (temf_arith_check).
__global__ void k_check_quotient(int n, const double* __restrict__ a, const double* __restrict__ b,
                                 double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double q = quotient(a[i], b[i], 1.0 / b[i]);
  out[i] = divisor_fits(b[i]) && quotient_key(q) >= kQuotientKey && isfinite(q) ? q : a[i] / b[i];
}
__global__ void k_check_dmma(int n, const double* __restrict__ a, const double* __restrict__ b,
                             double* __restrict__ out) {
  const int t = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32);
  if (t >= n) return;  // whole warps
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  double* c = out + 64 * (size_t)t + 8 * g + 2 * q;
  double c0 = c[0], c1 = c[1];
  dmma_8x8x4(c0, c1, a[32 * (size_t)t + 4 * g + q], b[32 * (size_t)t + 8 * q + g]);
  c[0] = c0;
  c[1] = c1;
}

void arith_check(int which, int n, const double* a, const double* b, double* out) {
  const size_t in = which == 0 ? n : 32 * (size_t)n, res = which == 0 ? n : 64 * (size_t)n;
  DBuf<double> da, db, dc;
  da.upload(a, in, 0);
  db.upload(b, in, 0);
  dc.upload(out, res, 0);
  if (which == 0) k_check_quotient<<<ceil_div(n, 256), 256>>>(n, da.p, db.p, dc.p);
  else k_check_dmma<<<ceil_div(32 * (int64_t)n, 256), 256>>>(n, da.p, db.p, dc.p);
  TEMF_CHECK_LAUNCH();
  TEMF_CUDA(cudaMemcpy(out, dc.p, res * sizeof(double), cudaMemcpyDeviceToHost));
}

// Bulk global -> shared copies on the TMA engine (cp.async.bulk, this GPU's
// own memory, each CTA its own copy), completed on an mbarrier: one instruction per
// panel column segment instead of one 8-byte copy per element.  Addresses
// and sizes must be multiples of 16 bytes: a segment that starts at an odd
// double is copied from one double earlier (its rows then start at offset 1
// of the shared row), and the size is rounded up to 16 bytes -- at most one
// double past the segment, which stays inside the slot allocation (the
// panels are followed by the scaled diagonal copies).
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const double* src, unsigned bytes, uint64_t* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(dst)),
               "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(b))
               : "memory");
}
// Bounded wait for a phase of the copy barrier: gives up after ~seconds and
// reports through the error word (the factor is then refused by the host).
constexpr int kCopySpinLimit = 1 << 22;
__device__ __forceinline__ void mbar_wait(uint64_t* b, unsigned parity, int* err) {
  for (int it = 0; !mbar_try_wait(b, parity); ++it) {
    if (it > kCopySpinLimit) {
      atomicExch(err, 1);
      return;
    }
    if (it > 64) __nanosleep(32);
  }
}

// Schur update tiles.  A tile (s, i0, j0, members m, column limit jl) holds
// C = sum over the m supernodes q = s-m+1 .. s of L21_q[rows beyond] *
// L21_q[rows beyond]^T for the kT x kT block (i0.., j0..) of s's row list:
// m > 1 for the column blocks of one wider supernode (a run), whose updates
// beyond the run are summed in one pass (K = the run's columns, each member's
// rows beyond the run are the rows of s, at offset r_q - r_s of its list);
// m = 1 otherwise.  jl > 0 restricts the tile to columns j < jl (inside a run,
// a member updates the later members' columns only).  C is scattered into the
// ancestors' panels through the relative indices of s, one red.global.add per
// entry (no read comes back to wait for; a level of several supernodes needs
// atomics anyway).  The K loop runs over 16-column chunks of the members
// through kStages buffers: bulk copies (one per column segment of A and of B:
// 32 per chunk, issued by warp 0) are in flight while the DMMA tiles consume
// the current chunk; the targets of the tile's columns are looked up
// meanwhile.
//
// Tile size and buffers go by the tiles launched together (update_shape).
// More than one wave of 64 x 64 tiles with four buffers (three CTAs per SM):
// two buffers and five CTAs per SM, bound by the FP64 tensor pipe (27k edges
// 1.58 ms a factorisation with the line at 3 tiles per SM, 1.62 at 8; 301k
// 19.0 and 19.1).  Up to one wave is bound by the latency of a tile, and four
// buffers hide the copies'.  Fewer tiles than SMs: 32 x 32 tiles, four times as
// many and a quarter as long (a tile of 512 columns on its own: 83 us with two
// buffers and a read-modify-write scatter, 49 as 32 x 32 tiles).  An entry's sum
// runs over the same columns in the same order in every shape.
constexpr int kUpdChunk = 16;

template <int kT, int kStages>
constexpr size_t update_smem() {
  return (size_t)kStages * 2 * kUpdChunk * (kT + 4) * sizeof(double);
}

template <int kT, int kStages>
__global__ void __launch_bounds__(128, kStages == 2 ? 5 : 3) k_update(
    const UpdTile* __restrict__ tiles, const int* __restrict__ sn_first,
    const int64_t* __restrict__ rows_ptr, const int* __restrict__ sn_rows,
    const int64_t* __restrict__ Lptr, const int* __restrict__ row_grp,
    const int* __restrict__ grp_target, const int* __restrict__ grp_shift,
    const int64_t* __restrict__ grp_relind, const int* __restrict__ relind, double* __restrict__ L,
    const double* __restrict__ sgn, int* __restrict__ err) {
  constexpr int kLd = kT + 4;   // fragment loads (4 columns x 8 rows) without bank conflicts; room for the shift
  constexpr int kF = kT / 16;   // 8-wide fragments per warp and side: warps 2 x 2 of kT/2 x kT/2
  extern __shared__ __align__(128) double sm[];
  __shared__ __align__(8) uint64_t mbar[kStages];
  __shared__ unsigned char shift[kStages][2][kUpdChunk];  // per buffer, operand, row: offset of the segment's first row
  __shared__ int64_t tcol[kT], trel[kT];                  // per column: its target column, its relative indices
  // [buffer][A | B][kUpdChunk][kLd]
  auto As = [&](int buf) { return sm + (size_t)buf * 2 * kUpdChunk * kLd; };
  auto Bs = [&](int buf) { return sm + (size_t)buf * 2 * kUpdChunk * kLd + kUpdChunk * kLd; };
  const UpdTile tile = tiles[blockIdx.x];
  const int s = tile.s;
  const int m = tile.mj & 15;
  const int jl = tile.mj >> 4;
  const int64_t rp = rows_ptr[s];
  const int r = (int)(rows_ptr[s + 1] - rp);
  const int tid = threadIdx.x;
  // K chunks of kUpdChunk columns over the members in order; a cursor
  // (member, first column) for the chunk being copied and one for the chunk
  // being multiplied
  int nch = 0;
  for (int u = 0; u < m; ++u) {
    const int q = s - m + 1 + u;
    nch += (sn_first[q + 1] - sn_first[q] + kUpdChunk - 1) / kUpdChunk;
  }
  int cp_q = s - m + 1, cp_k0 = 0, mm_q = s - m + 1, mm_k0 = 0;
  auto advance = [&](int& q, int& k0) {
    k0 += kUpdChunk;
    if (k0 >= sn_first[q + 1] - sn_first[q]) {
      ++q;
      k0 = 0;
    }
  };
  auto issue = [&](int buf) {  // warp 0
    const int q = cp_q, k0 = cp_k0;
    advance(cp_q, cp_k0);
    const int fq = sn_first[q];
    const int cq = sn_first[q + 1] - fq;
    const int rq = (int)(rows_ptr[q + 1] - rows_ptr[q]);
    const int64_t ldq = cq + rq;
    const double* P = L + Lptr[q] + cq + (rq - r);  // row 0 of the rows beyond the run
    // one segment per lane (operand A rows i0.., B rows j0..)
    const int op = tid / kUpdChunk, k = tid % kUpdChunk, kk = k0 + k;
    const int g0 = op == 0 ? tile.i0 : tile.j0;
    double* row = (op == 0 ? As(buf) : Bs(buf)) + k * kLd;
    if (kk < cq && g0 < r) {
      const double* src = P + (int64_t)kk * ldq + g0;
      const int n = min(kT, r - g0);  // rows past r only feed outputs that are not scattered
      const int o = (__cvta_generic_to_global(src) & 15) ? 1 : 0;
      const unsigned bytes = (unsigned)(((n + o) * 8 + 15) & ~15);
      shift[buf][op][k] = (unsigned char)o;
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      mbar_expect_tx(&mbar[buf], bytes);
      bulk_g2s(row, src - o, bytes, &mbar[buf]);
    } else {  // past the member's columns: a zero row
      shift[buf][op][k] = 0;
      for (int ii = 0; ii < kT; ++ii) row[ii] = 0.0;
    }
    __syncwarp();
    if (tid == 0) mbar_arrive(&mbar[buf]);
  };
  const int warp = tid >> 5, lane = tid & 31;
  const int wr = (warp >> 1) * (kT / 2), wc = (warp & 1) * (kT / 2);
  const int g = lane >> 2, qd = lane & 3;
  double acc[kF][kF][2];
#pragma unroll
  for (int a = 0; a < kF; ++a)
#pragma unroll
    for (int b = 0; b < kF; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  if (tid == 0) {
#pragma unroll
    for (int u = 0; u < kStages; ++u) mbar_init(&mbar[u], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int u = 0; u < kStages - 1; ++u)
      if (u < nch) issue(u);
  }
  // scatter targets of the tile's columns (read after the K loop's barriers)
  const int jend = jl > 0 ? min(jl, r) : r;
  if (tid >= 128 - kT) {
    const int jj = tid - (128 - kT), j = tile.j0 + jj;
    if (j < jend) {
      const int grp = row_grp[rp + j];
      const int t = grp_target[grp];
      const int ft = sn_first[t];
      const int64_t ldt = sn_first[t + 1] - ft + (rows_ptr[t + 1] - rows_ptr[t]);
      tcol[jj] = Lptr[t] + (int64_t)(sn_rows[rp + j] - ft) * ldt - grp_shift[grp];
      trel[jj] = grp_relind[grp];
    }
  }
  unsigned phases = 0u;  // bit b: parity of buffer b's next phase
  int buf = 0;
  for (int ch = 0; ch < nch; ++ch) {
    mbar_wait(&mbar[buf], (phases >> buf) & 1u, err);
    phases ^= 1u << buf;
    __syncthreads();  // the chunk before has been consumed: its buffer is free
    if (warp == 0 && ch + kStages - 1 < nch) issue(buf == 0 ? kStages - 1 : buf - 1);
    double* A = As(buf);
    const double* B = Bs(buf);
    if (sgn) {  // indefinite mode: A22 -= L21 S11 L21^T
      const int fq = sn_first[mm_q];
      const int cq = sn_first[mm_q + 1] - fq;
      for (int idx = tid; idx < kUpdChunk * kT; idx += blockDim.x) {
        const int k = idx / kT, ii = idx % kT;
        if (mm_k0 + k < cq) A[k * kLd + shift[buf][0][k] + ii] *= sgn[fq + mm_k0 + k];
      }
      __syncthreads();
      advance(mm_q, mm_k0);
    }
#pragma unroll 2
    for (int k0 = 0; k0 < kUpdChunk; k0 += 4) {
      double fa[kF], fb[kF];
      const int sa = shift[buf][0][k0 + qd], sb = shift[buf][1][k0 + qd];
#pragma unroll
      for (int a = 0; a < kF; ++a) fa[a] = A[(k0 + qd) * kLd + sa + wr + a * 8 + g];
#pragma unroll
      for (int b = 0; b < kF; ++b) fb[b] = B[(k0 + qd) * kLd + sb + wc + b * 8 + g];
#pragma unroll
      for (int a = 0; a < kF; ++a)
#pragma unroll
        for (int b = 0; b < kF; ++b) dmma_8x8x4(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
    }
    buf = buf == kStages - 1 ? 0 : buf + 1;
  }
  // scatter-subtract into the ancestors
#pragma unroll
  for (int b = 0; b < kF; ++b) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int jj = wc + b * 8 + 2 * qd + e, j = tile.j0 + jj;
      if (j >= jend) continue;
      double* dst = L + tcol[jj];
      const int* rel = relind + trel[jj];
      int at[kF];
#pragma unroll
      for (int a = 0; a < kF; ++a) {
        const int i = tile.i0 + wr + a * 8 + g;
        at[a] = i < r && i >= j ? rel[i] : -1;
      }
#pragma unroll
      for (int a = 0; a < kF; ++a)
        if (at[a] >= 0) atomicAdd(dst + at[a], -acc[a][b][e]);
    }
  }
}

// Shape of an update launch by its number of 64 x 64 tiles.
enum UpdShape { kUpdWide = 0, kUpdDeep = 1, kUpdSmall = 2 };
constexpr int kSms = 148;
inline UpdShape update_shape(int64_t tiles64) {
  return tiles64 > 3 * kSms ? kUpdWide : (tiles64 >= kSms ? kUpdDeep : kUpdSmall);
}

// ---------------------------------------------------------------------------
// host plan
// ---------------------------------------------------------------------------
void build_factor_plan(temf_ctx& c) {
  const Symbolic& S = c.sym;
  FactorPlan& F = c.fplan;
  cudaStream_t st = c.stream;
  F.sn_first.upload(S.sn_first.data(), S.sn_first.size(), st);
  F.sn_parent.upload(S.sn_parent.data(), S.sn_parent.size(), st);
  F.sn_rows.upload(S.sn_rows.data(), S.sn_rows.size(), st);
  F.sn_rows_ptr.upload(S.sn_rows_ptr.data(), S.sn_rows_ptr.size(), st);
  F.sn_Lptr.upload(S.sn_Lptr.data(), S.sn_Lptr.size(), st);
  F.level_sn.upload(S.level_sn.data(), S.level_sn.size(), st);
  F.level_ptr = S.level_ptr;

  auto width = [&](int s) { return S.sn_first[s + 1] - S.sn_first[s]; };
  auto nrows = [&](int s) { return (int64_t)(S.sn_rows_ptr[s + 1] - S.sn_rows_ptr[s]); };
  {  // the sweeps' scaled copies of the diagonal blocks, after the panels
    std::vector<int64_t> dp(S.nsn + 1);
    int64_t o = S.stored;
    for (int s = 0; s < S.nsn; ++s) {
      dp[s] = o;
      o += (int64_t)width(s) * width(s);
    }
    dp[S.nsn] = o;
    F.dsc_len = o - S.stored;
    F.dptr = dp;
    F.sn_Dptr.upload(F.dptr.data(), F.dptr.size(), st);
  }
  // position of global row i in the panel of supernode t (i >= first column of t)
  auto panel_row = [&](int t, int i) -> int64_t {
    const int ft = S.sn_first[t], ct = width(t);
    if (i < ft + ct) return i - ft;
    const int* b = S.sn_rows.data() + S.sn_rows_ptr[t];
    const int* e = S.sn_rows.data() + S.sn_rows_ptr[t + 1];
    const int* p = std::lower_bound(b, e, i);
    if (p == e || *p != i) throw StateError("symbolic structure inconsistent (row not in ancestor)");
    return ct + (p - b);
  };

  // A -> L map
  {
    std::vector<int> src;
    std::vector<int64_t> dst;
    const Pattern& P = c.pat;
    for (int i = 0; i < P.n; ++i) {
      for (int p = P.rowptr[i]; p < P.rowptr[i + 1]; ++p) {
        const int j = P.col[p];
        if (j > i) break;
        const int s = S.col2sn[j];
        const int64_t ld = width(s) + nrows(s);
        src.push_back(p);
        dst.push_back(S.sn_Lptr[s] + (int64_t)(j - S.sn_first[s]) * ld + panel_row(s, i));
      }
    }
    F.n_a2l = (int64_t)src.size();
    F.a2l_src.upload(src.data(), src.size(), st);
    F.a2l_dst.upload(dst.data(), dst.size(), st);
  }
  // update groups + relative indices (host threads; see symbolic.h)
  {
    UpdateGroups G;
    update_groups(S, G);
    F.n_relind = G.n_rel;
    F.row_grp.upload(G.row_grp.data(), G.row_grp.size(), st);
    F.grp_target.upload(G.grp_target.data(), G.grp_target.size(), st);
    F.grp_shift.upload(G.grp_shift.data(), G.grp_shift.size(), st);
    F.grp_relind.upload(G.grp_rel.data(), G.grp_rel.size(), st);
    F.relind.upload(G.rel.get(), (size_t)G.n_rel, st);
    TEMF_CUDA(cudaStreamSynchronize(st));  // G's host arrays go out of scope
  }
  // row chunks of the triangular solves per level
  {
    std::vector<TrsmChunk> ch;
    std::vector<int64_t> lp(S.nlevels + 1, 0);
    F.level_width.assign(S.nlevels, 0);
    for (int l = 0; l < S.nlevels; ++l) {
      for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; ++q) {
        const int s = S.level_sn[q];
        const int r = (int)nrows(s);
        for (int r0 = 0; r0 < r; r0 += kTrsmRows) ch.push_back({s, r0});
        F.level_width[l] = std::max(F.level_width[l], width(s));
      }
      lp[l + 1] = (int64_t)ch.size();
    }
    F.trsm_level_ptr = lp;
    F.n_trsm = (int64_t)ch.size();
    F.trsm.upload(reinterpret_cast<const int2*>(ch.data()), ch.size(), st);
  }
  // tiles per level, with runs of column blocks summed (see k_update)
  {
    const std::vector<int> run_end = update_runs(S, kUpdMaxMembers);
    F.n_runs = 0;
    std::vector<UpdTile> tiles;
    // tiles of level l with edge T appended
    auto level_tiles = [&](int l, int T, std::vector<UpdTile>& out, bool count_runs) {
      for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; ++q) {
        const int s = S.level_sn[q];
        const int r = (int)nrows(s);
        const int e = run_end[s];
        if (e != s) {
          // a run member before its last: only the later members' columns
          const int g = S.sn_first[e + 1] - S.sn_first[s + 1];
          for (int tj = 0; tj * T < g; ++tj)
            for (int ti = tj; ti * T < r; ++ti) out.push_back({s, ti * T, tj * T, 1 | (g << 4)});
          continue;
        }
        int m = 1;  // members of the run ending at s
        while (s - m >= 0 && run_end[s - m] == s) ++m;
        if (m > 1 && count_runs) ++F.n_runs;
        const int nt = ceil_div(r, T);
        for (int ti = 0; ti < nt; ++ti)
          for (int tj = 0; tj <= ti; ++tj) out.push_back({s, ti * T, tj * T, m});
      }
    };
    // A level's tiles in two parts: those with a column of the next level's
    // supernodes (the next level waits for them), then the others (by the 64
    // columns a tile lies in, whatever its own size).  One part where supernodes
    // of the level update entries in common: two parts run side by side, and the
    // one that arrives first decides the rounding of such an entry's sum.
    const std::vector<char> apart = levels_apart(S, run_end);
    int flagged = -1;  // supernode of `flags`: per 64 columns, whether they hold one
    std::vector<char> flags;
    auto urgent = [&](const UpdTile& t, int l) {
      if (t.s != flagged) {
        flagged = t.s;
        const int* rows = S.sn_rows.data() + S.sn_rows_ptr[t.s];
        const int r = (int)nrows(t.s), jl = t.mj >> 4, n = jl > 0 ? std::min(jl, r) : r;
        flags.assign(r / kUpdTile + 1, 0);
        for (int j = 0; j < n; ++j)
          if (S.sn_level[S.col2sn[rows[j]]] == l + 1) flags[j / kUpdTile] = 1;
      }
      return flags[t.j0 / kUpdTile] != 0;
    };
    F.upd.assign(2 * (size_t)S.nlevels, FactorPlan::UpdPart{});
    for (int l = 0; l < S.nlevels; ++l) {
      std::vector<UpdTile> all, small, part[2];
      level_tiles(l, kUpdTile, all, true);
      for (const UpdTile& t : all) part[!apart[l] || urgent(t, l) ? 0 : 1].push_back(t);
      for (int k = 0; k < 2; ++k) {
        FactorPlan::UpdPart& u = F.upd[2 * l + k];
        u.shape = update_shape((int64_t)part[k].size());
        if (u.shape == kUpdSmall && !part[k].empty()) {
          if (small.empty()) level_tiles(l, kUpdTile / 2, small, false);
          part[k].clear();
          for (const UpdTile& t : small)
            if ((!apart[l] || urgent(t, l)) == (k == 0)) part[k].push_back(t);
        }
        u.first = (int64_t)tiles.size();
        tiles.insert(tiles.end(), part[k].begin(), part[k].end());
        u.count = (int64_t)tiles.size() - u.first;
        if (u.count > INT_MAX) throw StateError("too many update tiles in one level");
      }
    }
    F.n_tiles = (int64_t)tiles.size();
    F.tiles.upload(tiles.data(), tiles.size(), st);
  }
  TEMF_CUDA(cudaStreamSynchronize(st));
}

int numeric_factor(temf_ctx& c, int slot, double dt) {
  // A(dt) = 0*A_eps + 3*M_sigma + 2*dt*K  (mkl_add_3 at src/FETD_FWD.f90:1288,1354)
  return numeric_factor_values(c, slot, c.d_M.p, 3.0, c.d_K.p, 2.0 * dt);
}

int numeric_factor_values(temf_ctx& c, int slot, const double* X, double a, const double* Y, double b) {
  launch_factor_values(c, slot, X, a, Y, b);
  return finish_factor(c, slot);
}

int numeric_factor_values_fallback(temf_ctx& c, int slot, const double* X, double a, const double* Y, double b) {
  const int st = numeric_factor_values(c, slot, X, a, Y, b);
  if (st <= 0) return st;
  // not positive definite: refactor in the indefinite mode (the reference
  // retries PARDISO with mtype -2, src/FETD_UTILITY.f90:923-935)
  launch_factor_values(c, slot, X, a, Y, b, true);
  finish_factor(c, slot);
  return st;
}

int finish_factor(temf_ctx& c, int slot) {
  FactorSlot& fs = c.slots[slot];
  int words[4] = {0, 0, 0, 0};
  TEMF_CUDA(cudaMemcpyAsync(words, c.d_status.p, 4 * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  TEMF_CUDA(cudaStreamSynchronize(c.stream));
  if (words[3] != 0) {
    fs.valid = false;
    throw StateError("a factor update's panel copies did not complete (bounded wait timed out)");
  }
  const int status = words[0];
  fs.perturbed = fs.indefinite ? words[2] : 0;
  if (status != INT_MAX) {
    // the first non-positive pivot (original numbering); an indefinite-mode
    // factor is valid nonetheless
    fs.status = c.sym.perm[status - 1] + 1;
    fs.valid = fs.indefinite;
    return fs.status;
  }
  fs.valid = true;
  fs.status = 0;
  return 0;
}

int64_t factor_launch_count(const temf_ctx& c) {
  const FactorPlan& F = c.fplan;
  int64_t n = F.n_a2l > 0 ? 1 : 0;
  for (int l = 0; l < c.sym.nlevels; ++l)
    n += (c.sym.level_ptr[l + 1] > c.sym.level_ptr[l]) + (F.trsm_level_ptr[l + 1] > F.trsm_level_ptr[l]) +
         (F.upd[2 * l].count > 0) + (F.upd[2 * l + 1].count > 0);
  return n;
}

void launch_factor(temf_ctx& c, int slot, double dt) {
  launch_factor_values(c, slot, c.d_M.p, 3.0, c.d_K.p, 2.0 * dt);
}

void launch_factor_values(temf_ctx& c, int slot, const double* X, double a, const double* Y, double b,
                          bool indefinite) {
  const Symbolic& S = c.sym;
  FactorPlan& F = c.fplan;
  FactorSlot& fs = c.slots[slot];
  cudaStream_t st = c.stream;
  fs.valid = false;
  if (fs.L.n < (size_t)slot_len(c)) fs.L.alloc(slot_len(c));
  TEMF_CUDA(cudaMemsetAsync(fs.L.p, 0, S.stored * sizeof(double), st));
  int init[3] = {INT_MAX, 0, 0};
  TEMF_CUDA(cudaMemcpyAsync(c.d_status.p, &init[0], sizeof(int), cudaMemcpyHostToDevice, st));
  TEMF_CUDA(cudaMemcpyAsync(c.d_status.p + 2, &init[2], sizeof(int), cudaMemcpyHostToDevice, st));
  TEMF_CUDA(cudaMemcpyAsync(c.d_status.p + 3, &init[1], sizeof(int), cudaMemcpyHostToDevice, st));  // copy waits
  fs.X = X;
  fs.a = a;
  fs.Y = Y;
  fs.b = b;
  fs.indefinite = indefinite;
  double* sgn = nullptr;
  if (indefinite) {
    if (fs.sgn.n < (size_t)S.n) fs.sgn.alloc(S.n);
    sgn = fs.sgn.p;
  }
  if (F.n_a2l) {
    k_load_A<<<ceil_div(F.n_a2l, 256), 256, 0, st>>>(F.n_a2l, F.a2l_src.p, F.a2l_dst.p, X, a, Y, b, fs.L.p);
    TEMF_CHECK_LAUNCH();
  }
  const auto upd_wide = k_update<kUpdTile, 2>;
  const auto upd_deep = k_update<kUpdTile, 4>;
  const auto upd_small = k_update<kUpdTile / 2, 4>;
  TEMF_CUDA(cudaFuncSetAttribute(upd_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)update_smem<kUpdTile, 2>()));
  TEMF_CUDA(cudaFuncSetAttribute(upd_deep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)update_smem<kUpdTile, 4>()));
  TEMF_CUDA(cudaFuncSetAttribute(k_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)trsm_smem(kSnCols)));
  const auto update = [&](const FactorPlan::UpdPart& u, cudaStream_t s) {
    if (u.count == 0) return;
    const auto upd = u.shape == kUpdWide ? upd_wide : (u.shape == kUpdDeep ? upd_deep : upd_small);
    const size_t smem = u.shape == kUpdWide ? update_smem<kUpdTile, 2>()
                                            : (u.shape == kUpdDeep ? update_smem<kUpdTile, 4>() : update_smem<kUpdTile / 2, 4>());
    upd<<<(unsigned)u.count, 128, smem, s>>>(F.tiles.p + u.first, F.sn_first.p, F.sn_rows_ptr.p, F.sn_rows.p,
                                             F.sn_Lptr.p, F.row_grp.p, F.grp_target.p, F.grp_shift.p, F.grp_relind.p,
                                             F.relind.p, fs.L.p, sgn, c.d_status.p + 3);
    TEMF_CHECK_LAUNCH();
  };
  // Two streams.  The chain (a level's blocks, its row solves, the updates
  // the next level waits for) runs on a high-priority stream, the level's
  // other updates on the context's stream, behind the next level's blocks and
  // row solves (one CTA and a few, about 30 us).  A level's urgent updates
  // wait for the other updates of the level before, and the two parts of a
  // level have no entry in common (levels_apart): every entry receives its
  // sums as in one stream.
  FactorStreams& W = c.fac;
  W.ensure();
  const cudaStream_t hi = W.chain;
  TEMF_CUDA(cudaEventRecord(W.chain_at, st));
  TEMF_CUDA(cudaStreamWaitEvent(hi, W.chain_at, 0));
  // whatever ends the loop, the context's stream comes after what the chain runs
  struct Join {
    FactorStreams& W;
    cudaStream_t st;
    ~Join() {
      cudaEventRecord(W.chain_at, W.chain);
      cudaStreamWaitEvent(st, W.chain_at, 0);
    }
  } join{W, st};
  bool rest_pending = false;  // updates on st that the chain has not waited for
  for (int l = 0; l < S.nlevels; ++l) {
    const int cnt = S.level_ptr[l + 1] - S.level_ptr[l];
    if (cnt > 0) {
      const auto potrf = indefinite ? k_potrf<true> : k_potrf<false>;
      potrf<<<cnt, kPotrfThreads, 0, hi>>>(F.level_sn.p + S.level_ptr[l], F.sn_first.p, F.sn_rows_ptr.p, F.sn_Lptr.p,
                                           fs.L.p, c.d_status.p, sgn, F.sn_Dptr.p);
      TEMF_CHECK_LAUNCH();
    }
    const int64_t c0 = F.trsm_level_ptr[l], c1 = F.trsm_level_ptr[l + 1];
    if (c1 > c0) {
      k_trsm<<<(unsigned)(c1 - c0), kTrsmThreads, trsm_smem(F.level_width[l]), hi>>>(
          reinterpret_cast<const TrsmChunk*>(F.trsm.p) + c0, F.sn_first.p, F.sn_rows_ptr.p, F.sn_Lptr.p, fs.L.p, sgn);
      TEMF_CHECK_LAUNCH();
    }
    const FactorPlan::UpdPart &now = F.upd[2 * l], &rest = F.upd[2 * l + 1];
    if (rest.count) TEMF_CUDA(cudaEventRecord(W.chain_at, hi));
    if (rest_pending) {
      TEMF_CUDA(cudaStreamWaitEvent(hi, W.rest_at, 0));
      rest_pending = false;
    }
    update(now, hi);
    if (rest.count) {
      TEMF_CUDA(cudaStreamWaitEvent(st, W.chain_at, 0));
      update(rest, st);
      TEMF_CUDA(cudaEventRecord(W.rest_at, st));
      rest_pending = true;
    }
  }
  fs.dt = b * 0.5;
}

}  // namespace temf
