// precond.cu -- the leaf-block-diagonal preconditioner (LEAFMATVECpara,
// treecode3d_pb.f:1393-1542) and the diagonal one (MSOLVEprec, main.f90:532-542).
//
// Per leaf of n faces the reference assembles the 2n x 2n column-major block
//   row i, col j      : -A_j (G1 - eps G2)      (j != i)       = -A_j K1
//   row i+n, col j    : -A_j (G0 - Gk)                         = -A_j K2
//   row i, col j+n    : -A_j (G4 - G3)                         = -A_j K3
//   row i+n, col j+n  : -A_j (G10 - G20/eps)                   = -A_j K4
//   diagonal          : pre1 (rows 1..n), pre2 (rows n+1..2n)
// (K2 and K3 sit in the transposed block positions relative to the matvec
// operator -- reproduced as is), then calls DGETRF (which, with the vendored
// testing ILAENV, is the unblocked recursive DGETRF2: partial pivoting on the
// largest |a|, first index on ties) and DGETRS, on EVERY call.  The block
// never changes, so here it is assembled and factored once per tree
// (right-looking LU with partial pivoting, the same pivot rule, batched over
// all leaves) and every apply is a blocked forward/back substitution.
#include <algorithm>
#include <optional>
#include <climits>

#include "fast_math.cuh"
#include "tabi_impl.cuh"

namespace tabi {

namespace {

constexpr int kAsmCols = 8;

// CHECK false: kappa times the distance is inside the exponential's table.
// The four kernels of one pair times -A_j (d = r_j - r_i, m = A_j v_j; the near
// field's forms, see matvec.cu), 1/(4 pi) included in A_j.
template <bool CHECK>
__device__ __forceinline__ void asm_pair(double dx, double dy, double dz, double vx, double vy,
                                         double vz, double mx, double my, double mz, double A,
                                         double kappa, double eps, double inv_eps,
                                         const double* tab, double& K1, double& K2, double& K3,
                                         double& K4) {
  const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
  const double i = fast_rsqrt(r2), i2 = i * i, i3 = i * i2;
  const double kr = kappa * (r2 * i);
  const double e = exp_neg<CHECK>(kr, tab);
  const double t = fma(kr, e, e);
  const double md = fma(mx, dx, fma(my, dy, mz * dz));
  const double vd = fma(vx, dx, fma(vy, dy, vz * dz));
  const double mv = fma(mx, vx, fma(my, vy, mz * vz));
  const double mvd = md * vd;
  K1 = -(i3 * md) * fma(-eps, t, 1.0);
  K2 = -(i * A) * (1.0 - e);
  K3 = -i3 * fma(-(kappa * kappa) * e, mvd, fma(-3.0 * i2, mvd, mv) * (t - 1.0));
  K4 = -(i3 * A) * vd * fma(-inv_eps, t, 1.0);
}

// One block per (leaf, 8 columns), tiles given as (leaf, j0).  A warp takes 32
// rows of one column at a time, so that leaves of any size keep the block's
// warps busy (with a thread per row the mean leaf of 160 left 96 of 256
// idle).
template <bool CHECK>
__global__ void __launch_bounds__(256) assemble_kernel(
    const int2* __restrict__ tiles, const int2* __restrict__ leaf_rng,
    const int64_t* __restrict__ blk_off, const double* __restrict__ px,
    const double* __restrict__ py, const double* __restrict__ pz, const double* __restrict__ nx,
    const double* __restrict__ ny, const double* __restrict__ nz,
    const double* __restrict__ area, double kappa, double eps, double* __restrict__ lu) {
  __shared__ double tab[kExpTab];
  exp_table_fill(tab);
  __syncthreads();
  const int2 tl = tiles[blockIdx.x];
  const int2 lr = leaf_rng[tl.x];
  const int ib = lr.x, n = lr.y, m = 2 * n;
  double* A = lu + blk_off[tl.x];
  const double pre1 = 0.5 * (1.0 + eps), pre2 = 0.5 * (1.0 + 1.0 / eps);
  const double inv_eps = 1.0 / eps;
  const int lane = threadIdx.x & 31, cols = min(kAsmCols, n - tl.y);
  for (int q = threadIdx.x >> 5; q < cols * ((n + 31) >> 5); q += 8) {
    const int j = tl.y + q % cols, i = 32 * (q / cols) + lane;
    if (i >= n) continue;
    double* c1 = A + (size_t)j * m;        // column j
    double* c2 = A + (size_t)(j + n) * m;  // column j + n
    double K1 = pre1, K2 = 0.0, K3 = 0.0, K4 = pre2;
    if (i != j) {
      const int t = ib + i, s = ib + j;
      const double Aj = area[s] * kOneOver4Pi;
      asm_pair<CHECK>(px[s] - px[t], py[s] - py[t], pz[s] - pz[t], nx[t], ny[t], nz[t], Aj * nx[s],
               Aj * ny[s], Aj * nz[s], Aj, kappa, eps, inv_eps, tab, K1, K2, K3, K4);
    }
    c1[i] = K1;
    c1[i + n] = K2;
    c2[i] = K3;
    c2[i + n] = K4;
  }
}

constexpr int kLuThreads = 256;
constexpr int kNB = 32;   // panel width
constexpr int kTM = 64;   // trailing-update tile

__device__ __forceinline__ void argmax_merge(double& v, int& i, double v2, int i2) {
  if (v2 > v || (v2 == v && i2 < i)) {
    v = v2;
    i = i2;
  }
}

// Right-looking blocked LU with partial pivoting of one leaf block per CTA,
// panel in global memory (used for blocks too large for the shared-memory
// panel of the batched kernels).
__global__ void __launch_bounds__(kLuThreads) lu_kernel(const int* __restrict__ leaves,
                                                        const int2* __restrict__ leaf_rng,
                                                        const int64_t* __restrict__ blk_off,
                                                        double* __restrict__ lu,
                                                        int* __restrict__ piv,
                                                        int* __restrict__ info,
                                                        int skip_max_m) {
  int leaf = leaves[blockIdx.x];
  int2 lr = leaf_rng[leaf];
  int m = 2 * lr.y;
  if (m <= skip_max_m) return;  // factored by the batched kernels
  double* A = lu + blk_off[leaf];
  int* ip = piv + 2 * lr.x;
  __shared__ double s_v[kLuThreads / 32];
  __shared__ int s_i[kLuThreads / 32];
  __shared__ int s_p;
  __shared__ double sL[kTM][kNB + 1];
  __shared__ double sU[kNB][kTM + 1];
  int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int my_info = 0;
  for (int k0 = 0; k0 < m; k0 += kNB) {
    int nb = min(kNB, m - k0);
    // ---- panel factorization (columns k0 .. k0+nb-1)
    for (int kk = k0; kk < k0 + nb; ++kk) {
      double* col = A + (size_t)kk * m;
      // a column of NaNs offers no candidate: the diagonal row stays the pivot
      double bv = -1.0;
      int bi = kk;
      for (int i = kk + tid; i < m; i += blockDim.x) argmax_merge(bv, bi, fabs(col[i]), i);
      for (int o = 16; o > 0; o >>= 1) {
        double v2 = __shfl_xor_sync(0xffffffffu, bv, o);
        int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
        argmax_merge(bv, bi, v2, i2);
      }
      if (lane == 0) {
        s_v[warp] = bv;
        s_i[warp] = bi;
      }
      __syncthreads();
      if (tid == 0) {
        double v = s_v[0];
        int i = s_i[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) argmax_merge(v, i, s_v[w], s_i[w]);
        s_p = i;
        ip[kk] = i + 1;  // 1-based like LAPACK
      }
      __syncthreads();
      int p = s_p;
      double pv = col[p];
      if (pv == 0.0) {
        if (my_info == 0) my_info = kk + 1;
        __syncthreads();
        continue;  // DGETRF2: no swap, no scaling, INFO set
      }
      if (p != kk)
        for (int c = tid; c < m; c += blockDim.x) {
          double* cc = A + (size_t)c * m;
          double t = cc[kk];
          cc[kk] = cc[p];
          cc[p] = t;
        }
      __syncthreads();
      pv = col[kk];
      if (fabs(pv) >= 2.2250738585072014e-308) {
        double r = 1.0 / pv;
        for (int i = kk + 1 + tid; i < m; i += blockDim.x) col[i] *= r;
      } else {
        for (int i = kk + 1 + tid; i < m; i += blockDim.x) col[i] /= pv;
      }
      __syncthreads();
      // rank-1 update of the rest of the panel
      int ncol = k0 + nb - kk - 1;
      int nrow = m - kk - 1;
      for (int q = tid; q < ncol * nrow; q += blockDim.x) {
        int c = kk + 1 + q / nrow;
        int i = kk + 1 + q % nrow;
        double* cc = A + (size_t)c * m;
        cc[i] = fma(-col[i], cc[kk], cc[i]);
      }
      __syncthreads();
    }
    int c1 = k0 + nb;
    if (c1 >= m) break;
    // ---- U12 = L11^{-1} A12 (unit lower), one column per thread
    for (int c = c1 + tid; c < m; c += blockDim.x) {
      double* cc = A + (size_t)c * m;
      double xv[kNB];
#pragma unroll
      for (int r = 0; r < kNB; ++r) xv[r] = (r < nb) ? cc[k0 + r] : 0.0;
#pragma unroll
      for (int r = 1; r < kNB; ++r) {
        if (r < nb) {
          double s = xv[r];
#pragma unroll
          for (int q = 0; q < kNB; ++q)
            if (q < r) s = fma(-A[(size_t)(k0 + q) * m + k0 + r], xv[q], s);
          xv[r] = s;
        }
      }
#pragma unroll
      for (int r = 0; r < kNB; ++r)
        if (r < nb) cc[k0 + r] = xv[r];
    }
    __syncthreads();
    // ---- A22 -= L21 * U12, 64x64 tiles, 4x4 per thread
    int rows = m - c1;
    int ntr = (rows + kTM - 1) / kTM;
    int tr = tid / 16, tc = tid % 16;  // 16 x 16 thread grid
    for (int tile = 0; tile < ntr * ntr; ++tile) {
      int r0 = c1 + (tile / ntr) * kTM;
      int cb = c1 + (tile % ntr) * kTM;
      // load L21 tile (kTM x nb) and U12 tile (nb x kTM)
      for (int q = tid; q < kTM * kNB; q += blockDim.x) {
        int r = q % kTM, k = q / kTM;
        int gr = r0 + r;
        sL[r][k] = (gr < m && k < nb) ? A[(size_t)(k0 + k) * m + gr] : 0.0;
      }
      for (int q = tid; q < kNB * kTM; q += blockDim.x) {
        int k = q % kNB, c = q / kNB;
        int gc = cb + c;
        sU[k][c] = (gc < m && k < nb) ? A[(size_t)gc * m + k0 + k] : 0.0;
      }
      __syncthreads();
      double acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
#pragma unroll 8
      for (int k = 0; k < kNB; ++k) {
        double lv[4], uv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) lv[a] = sL[tr + 16 * a][k];
#pragma unroll
        for (int b = 0; b < 4; ++b) uv[b] = sU[k][tc + 16 * b];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[a][b] = fma(lv[a], uv[b], acc[a][b]);
      }
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        int gc = cb + tc + 16 * b;
        if (gc >= m) continue;
        double* cc = A + (size_t)gc * m;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          int gr = r0 + tr + 16 * a;
          if (gr < m) cc[gr] -= acc[a][b];
        }
      }
      __syncthreads();
    }
  }
  if (tid == 0) info[leaf] = my_info;
}


// Batched, level-synchronous right-looking LU with partial pivoting for all
// leaf blocks of order m <= kPanelMaxM at once, in outer blocks of kOB columns
// (the plan is built in build_precond).  Inside an outer block, panel step s
// (k0 = 32 s) is three launches over every block that still has columns left:
//   lu_panel_reg_kernel / lu_panel_kernel  one CTA per block: the 32-column
//                    panel (rows k0..m-1) as two 16-column halves -- pivot
//                    search (largest |a|, first index on ties, as IDAMAX), row
//                    swap, scaling, rank-1 updates; the second half first takes
//                    the first half's swaps, TRSM and GEMM update (DGETRF2's
//                    recursion, one level);
//   lu_strip_kernel  one CTA per 128-column strip of the outer block: the
//                    panel's row swaps, and for strips right of the panel
//                    U12 = L11^{-1} A12; strips left of the panel only take
//                    swaps (LAPACK applies every pivot to the L columns too);
//   lu_gemm_kernel   one CTA per 64 x 64 tile of the outer block right of the
//                    panel: A22 -= L21 U12 with k = 32.
// After the outer block, its row interchanges reach the columns left and right
// of it at once (lu_swapmap_kernel + lu_rowswap_kernel), U12 of the columns
// right of it follows by 32-row TRSM + small GEMM steps, and the trailing
// matrix takes one kOB-deep lu_gemm_kernel update.  The trailing updates of
// all blocks run concurrently across the GPU.
constexpr int kBP = 32;            // panel width
constexpr int kSP = 16;            // panel half held in shared memory
constexpr int kPanelMaxM = 1536;   // half panel of 1536 x 16 doubles = 192 KB
constexpr int kPT = 256;           // panel kernel threads
constexpr int kUT = 256;           // strip / gemm kernel threads
constexpr int kUC = 128;           // strip width
constexpr int kGT = 64;            // gemm tile
constexpr int kOB = 256;           // outer block: columns right of it are updated once per block
constexpr int kLuSmallBlock = 512; // blocks up to this order factor on the side stream

// Factor columns [c0l, c0l + nb) of the panel held in P (local column c of
// the half is P + c * mr, local row r = global row k0 + r) starting at local
// row r0; records 1-based global pivots.
__device__ void panel_factor(double* P, int mr, int r0, int nb, int k0, int* ip, int* info,
                             int leaf, double* s_v, int* s_i, int* s_p) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int j = 0; j < nb; ++j) {
    const int lr0 = r0 + j;  // local row of the diagonal
    double* col = P + (size_t)j * mr;
    // a column of NaNs offers no candidate: the diagonal row stays the pivot
    double bv = -1.0;
    int bi = lr0;
    for (int i = lr0 + tid; i < mr; i += kPT) argmax_merge(bv, bi, fabs(col[i]), i);
    for (int o = 16; o > 0; o >>= 1) {
      double v2 = __shfl_xor_sync(0xffffffffu, bv, o);
      int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
      argmax_merge(bv, bi, v2, i2);
    }
    if (lane == 0) {
      s_v[warp] = bv;
      s_i[warp] = bi;
    }
    __syncthreads();
    if (warp == 0) {
      double v = (lane < kPT / 32) ? s_v[lane] : -1.0;
      int i = (lane < kPT / 32) ? s_i[lane] : mr;
      for (int o = 16; o > 0; o >>= 1) {
        double v2 = __shfl_xor_sync(0xffffffffu, v, o);
        int i2 = __shfl_xor_sync(0xffffffffu, i, o);
        argmax_merge(v, i, v2, i2);
      }
      if (lane == 0) *s_p = i;
    }
    __syncthreads();
    const int p = *s_p;
    const double pv = col[p];
    if (pv == 0.0) {  // DGETRF2: INFO set, no swap, no scaling
      if (tid == 0) {
        atomicCAS(&info[leaf], 0, k0 + lr0 + 1);
        ip[k0 + lr0] = k0 + lr0 + 1;
      }
      __syncthreads();
      continue;
    }
    if (tid == 0) ip[k0 + lr0] = k0 + p + 1;  // 1-based, like LAPACK
    if (p != lr0 && tid < nb) {
      double* cc = P + (size_t)tid * mr;
      double t = cc[lr0];
      cc[lr0] = cc[p];
      cc[p] = t;
    }
    __syncthreads();
    const double pk = col[lr0];
    const bool recip = fabs(pk) >= 2.2250738585072014e-308;
    const double rcp = 1.0 / pk;
    for (int i = lr0 + 1 + tid; i < mr; i += kPT) {
      double l = recip ? col[i] * rcp : col[i] / pk;
      col[i] = l;
      for (int c = j + 1; c < nb; ++c) {
        double* cc = P + (size_t)c * mr;
        cc[i] = fma(-l, cc[lr0], cc[i]);
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kPT) lu_panel_kernel(const int* __restrict__ items, int k0,
                                                       const int2* __restrict__ leaf_rng,
                                                       const int64_t* __restrict__ blk_off,
                                                       double* __restrict__ lu,
                                                       int* __restrict__ piv,
                                                       int* __restrict__ info) {
  extern __shared__ double P[];
  __shared__ double s_v[kPT / 32];
  __shared__ int s_i[kPT / 32];
  __shared__ int s_p;
  __shared__ double sL11[kSP][kSP + 1];
  __shared__ int s_rows[2 * kSP], s_src[2 * kSP];
  const int leaf = items[blockIdx.x];
  const int2 lr = leaf_rng[leaf];
  const int m = 2 * lr.y;
  const int nb = min(kBP, m - k0), mr = m - k0;
  const int nb1 = min(kSP, nb), nb2 = nb - nb1;
  double* A = lu + blk_off[leaf];
  int* ip = piv + 2 * lr.x;
  const int tid = threadIdx.x;
  // ---- first half
  for (int q = tid; q < nb1 * mr; q += kPT) {
    int c = q / mr, r = q - c * mr;
    P[q] = A[(size_t)(k0 + c) * m + k0 + r];
  }
  __syncthreads();
  panel_factor(P, mr, 0, nb1, k0, ip, info, leaf, s_v, s_i, &s_p);
  for (int q = tid; q < nb1 * mr; q += kPT) {
    int c = q / mr, r = q - c * mr;
    A[(size_t)(k0 + c) * m + k0 + r] = P[q];
  }
  if (nb2 == 0) return;
  for (int q = tid; q < nb1 * nb1; q += kPT) {
    int c = q / nb1, r = q - c * nb1;
    sL11[r][c] = P[(size_t)c * mr + r];
  }
  __syncthreads();
  // ---- second half: load, first half's swaps, TRSM, GEMM update, factor
  const int c2 = k0 + kSP;
  for (int q = tid; q < nb2 * mr; q += kPT) {
    int c = q / mr, r = q - c * mr;
    P[q] = A[(size_t)(c2 + c) * m + k0 + r];
  }
  __syncthreads();
  if (tid < nb2) {
    double* cc = P + (size_t)tid * mr;
    for (int j = 0; j < nb1; ++j) {
      int p = ip[k0 + j] - 1 - k0;
      if (p != j) {
        double t = cc[j];
        cc[j] = cc[p];
        cc[p] = t;
      }
    }
    double x[kSP];
#pragma unroll
    for (int r = 0; r < kSP; ++r) x[r] = (r < nb1) ? cc[r] : 0.0;
#pragma unroll
    for (int r = 1; r < kSP; ++r) {
      double acc = x[r];
#pragma unroll
      for (int q = 0; q < kSP; ++q)
        if (q < r) acc = fma(-sL11[r][q], x[q], acc);
      x[r] = acc;
    }
#pragma unroll
    for (int r = 0; r < kSP; ++r)
      if (r < nb1) cc[r] = x[r];
  }
  __syncthreads();
  // rows kSP.. of the second half -= L21 (first half, global) * U (rows 0..15 of P)
  for (int i = kSP + tid; i < mr; i += kPT) {
    double l[kSP];
#pragma unroll
    for (int q = 0; q < kSP; ++q) l[q] = A[(size_t)(k0 + q) * m + k0 + i];
    for (int c = 0; c < nb2; ++c) {
      double* cc = P + (size_t)c * mr;
      double acc = cc[i];
#pragma unroll
      for (int q = 0; q < kSP; ++q) acc = fma(-l[q], cc[q], acc);
      cc[i] = acc;
    }
  }
  __syncthreads();
  panel_factor(P, mr, kSP, nb2, k0, ip, info, leaf, s_v, s_i, &s_p);
  for (int q = tid; q < nb2 * mr; q += kPT) {
    int c = q / mr, r = q - c * mr;
    A[(size_t)(c2 + c) * m + k0 + r] = P[q];
  }
  // the second half's swaps on the first half's columns (gathered through
  // shared memory: rows touched and, for each, the row its value comes from)
  __syncthreads();
  if (tid == 0) {
    int nr = 0;
    for (int j = kSP; j < nb; ++j) s_rows[nr++] = k0 + j;
    for (int j = kSP; j < nb; ++j) {
      int p = ip[k0 + j] - 1;
      bool have = false;
      for (int q = 0; q < nr; ++q) have |= (s_rows[q] == p);
      if (!have) s_rows[nr++] = p;
    }
    for (int q = 0; q < nr; ++q) s_src[q] = s_rows[q];
    for (int j = kSP; j < nb; ++j) {
      int p = ip[k0 + j] - 1, a = -1, b = -1;
      for (int q = 0; q < nr; ++q) {
        if (s_rows[q] == k0 + j) a = q;
        if (s_rows[q] == p) b = q;
      }
      int t = s_src[a];
      s_src[a] = s_src[b];
      s_src[b] = t;
    }
    s_p = nr;
  }
  __syncthreads();
  const int nr = s_p;
  for (int q = tid; q < nr * nb1; q += kPT) {
    int row = q / nb1, c = q - row * nb1;
    P[q] = A[(size_t)(k0 + c) * m + s_src[row]];
  }
  __syncthreads();
  for (int q = tid; q < nr * nb1; q += kPT) {
    int row = q / nb1, c = q - row * nb1;
    A[(size_t)(k0 + c) * m + s_rows[row]] = P[q];
  }
}

// The same panel step with the panel half held in registers: thread t owns
// the local rows t + NT q (q < R), all 16 columns of the half.  Per column a
// single CTA barrier: before it, every warp publishes its best candidate
// (|value|, row) and that row's 16 values, and the owner of the diagonal row
// publishes it; after it, every warp reduces the candidates itself, takes the
// winner's row as the pivot row, and each thread swaps, scales and updates its
// own rows.  Candidates are double-buffered by step parity, so a fast warp's
// writes of step j+1 cannot meet a slow warp's reads of step j.  The column
// in work is always register 0: after each step a thread rotates its rows'
// 16 registers left by one, so the column loop needs no unrolling (an
// unrolled loop overflowed the instruction cache) and after 16 steps the
// registers are back in column order.  The operations and their order equal
// lu_panel_kernel's, so the factors are the same bit for bit.
constexpr int kRegMaxRows = 2;  // rows per thread of the register panel

struct PanelShared {
  static constexpr int kMaxW = 16;
  double cand[2][kMaxW][kSP];  // each warp's best row (rotated order)
  double cv[2][kMaxW];         // its |value|
  int ci[2][kMaxW];            // its local row
  double lrow[2][kSP];         // the diagonal row before the swap
  int piv[kBP];                // local pivot rows of the panel's columns
  double u12[kSP][kSP + 1];    // second half: U12 after the TRSM
};

template <int NT, int R>
__device__ __forceinline__ void panel_half_reg(double (&a)[R][kSP], int mr, int rbase, int nbh,
                                               int k0, int& st, int* ip, int* info, int leaf,
                                               PanelShared& S) {
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll 1
  for (int j = 0; j < kSP; ++j) {  // nbh pivot steps, then rotations only
    if (j < nbh) {                 // uniform over the CTA
      const int lr0 = rbase + j, b = st & 1, rem = nbh - j;
      double bv = -1.0;
      int bi = INT_MAX;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int r = tid + NT * q;
        if (r >= lr0 && r < mr) argmax_merge(bv, bi, fabs(a[q][0]), r);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double v2 = __shfl_xor_sync(0xffffffffu, bv, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
        argmax_merge(bv, bi, v2, i2);
      }
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int r = tid + NT * q;
        if (r == bi) {
#pragma unroll
          for (int c = 0; c < kSP; ++c) S.cand[b][warp][c] = a[q][c];
        }
        if (r == lr0) {
#pragma unroll
          for (int c = 0; c < kSP; ++c) S.lrow[b][c] = a[q][c];
        }
      }
      if (lane == 0) {
        S.cv[b][warp] = bv;
        S.ci[b][warp] = bi;
      }
      __syncthreads();
      double v = lane < NW ? S.cv[b][lane] : -1.0;
      int p = lane < NW ? S.ci[b][lane] : INT_MAX;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double v2 = __shfl_xor_sync(0xffffffffu, v, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, p, o);
        argmax_merge(v, p, v2, i2);
      }
      // no candidate at all (a column of NaNs): keep the diagonal row
      const double* urow = p == INT_MAX ? S.lrow[b] : S.cand[b][(p % NT) >> 5];
      if (p == INT_MAX) p = lr0;
      const double pv = urow[0];
      if (pv == 0.0) p = lr0;  // a zero column: no interchange
      if (tid == 0) {
        S.piv[lr0] = p;
        ip[k0 + lr0] = k0 + p + 1;  // 1-based, like LAPACK
      }
      if (pv != 0.0) {
        const bool recip = fabs(pv) >= 2.2250738585072014e-308;
        const double rcp = 1.0 / pv;
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const int r = tid + NT * q;
          if (p != lr0) {
            if (r == p) {
#pragma unroll
              for (int c = 0; c < kSP; ++c) a[q][c] = S.lrow[b][c];
            } else if (r == lr0) {
#pragma unroll
              for (int c = 0; c < kSP; ++c) a[q][c] = urow[c];
            }
          }
          if (r > lr0 && r < mr) {
            const double l = recip ? a[q][0] * rcp : a[q][0] / pv;
            a[q][0] = l;
#pragma unroll
            for (int c = 1; c < kSP; ++c)
              if (c < rem) a[q][c] = fma(-l, urow[c], a[q][c]);
          }
        }
      } else if (tid == 0) {  // DGETRF2: INFO set, no swap, no scaling
        atomicCAS(&info[leaf], 0, k0 + lr0 + 1);
      }
      ++st;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const double t0 = a[q][0];
#pragma unroll
      for (int c = 0; c < kSP - 1; ++c) a[q][c] = a[q][c + 1];
      a[q][kSP - 1] = t0;
    }
  }
}

// Source row of local row r after the row interchanges (j, piv[j]) for
// j = j0 .. j1-1 were applied in order: the swaps replayed backwards.
__device__ __forceinline__ int swapped_source(int r, const int* piv, int j0, int j1) {
  for (int j = j1 - 1; j >= j0; --j) {
    const int pj = piv[j];
    if (r == j) r = pj;
    else if (r == pj) r = j;
  }
  return r;
}

template <int NT, int R>
__global__ void __launch_bounds__(NT, 512 / NT) lu_panel_reg_kernel(
    const int* __restrict__ items, int k0, const int2* __restrict__ leaf_rng,
    const int64_t* __restrict__ blk_off, double* __restrict__ lu, int* __restrict__ piv,
    int* __restrict__ info) {
  static_assert(NT / 32 <= PanelShared::kMaxW, "too many warps");
  __shared__ PanelShared S;
  const int leaf = items[blockIdx.x];
  const int2 lr = leaf_rng[leaf];
  const int m = 2 * lr.y;
  const int nb = min(kBP, m - k0), mr = m - k0;
  const int nb1 = min(kSP, nb), nb2 = nb - nb1;
  double* A = lu + blk_off[leaf];
  int* ip = piv + 2 * lr.x;
  const int tid = threadIdx.x;
  int st = 0;
  double a[R][kSP];
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {  // the two 16-column halves
    const int nbh = h == 0 ? nb1 : nb2, cb = k0 + kSP * h;
    if (nbh == 0) break;
    if (h == 0) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int r = tid + NT * q;
#pragma unroll
        for (int c = 0; c < kSP; ++c)
          a[q][c] = (r < mr && c < nb1) ? A[(size_t)(k0 + c) * m + k0 + r] : 0.0;
      }
    } else {
      // load through the first half's swaps, TRSM, GEMM update
      __syncthreads();  // pivots and the stored first half visible to all
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int r = tid + NT * q;
        const int src = r < mr ? swapped_source(r, S.piv, 0, kSP) : r;
#pragma unroll
        for (int c = 0; c < kSP; ++c)
          a[q][c] = (r < mr && c < nb2) ? A[(size_t)(cb + c) * m + k0 + src] : 0.0;
      }
      if (tid < 32) {  // U12 = L11^{-1} A12: rows 0..15 are lanes 0..15, q = 0
        const int lane = tid;
        double l11[kSP];
#pragma unroll
        for (int q = 0; q < kSP; ++q)
          l11[q] = lane < kSP ? A[(size_t)(k0 + q) * m + k0 + lane] : 0.0;
#pragma unroll
        for (int q = 0; q < kSP - 1; ++q)
#pragma unroll
          for (int c = 0; c < kSP; ++c) {
            const double x = __shfl_sync(0xffffffffu, a[0][c], q);
            if (lane > q && lane < kSP) a[0][c] = fma(-l11[q], x, a[0][c]);
          }
        if (lane < kSP)
#pragma unroll
          for (int c = 0; c < kSP; ++c) S.u12[lane][c] = a[0][c];
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < R; ++q) {  // rows 16.. -= L21 U12 (per element k = 0..15 in order)
        const int r = tid + NT * q;
        if (r >= kSP && r < mr) {
          const double* lrow = A + (size_t)k0 * m + k0 + r;
#pragma unroll 1
          for (int k = 0; k < kSP; ++k) {
            const double l = lrow[(size_t)k * m];
#pragma unroll
            for (int c = 0; c < kSP; ++c) a[q][c] = fma(-l, S.u12[k][c], a[q][c]);
          }
        }
      }
    }
    panel_half_reg<NT, R>(a, mr, kSP * h, nbh, k0, st, ip, info, leaf, S);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int r = tid + NT * q;
      if (r < mr) {
#pragma unroll
        for (int c = 0; c < kSP; ++c)
          if (c < nbh) A[(size_t)(cb + c) * m + k0 + r] = a[q][c];
      }
    }
  }
  if (nb2 == 0) return;
  __syncthreads();
  // the second half's swaps on the first half's columns: slot s < 16 is the
  // diagonal row 16 + s, slot 16 + j the pivot row of column 16 + j when it is
  // below the panel's diagonal rows and not named by an earlier column
  constexpr int kPer = (2 * kSP * kSP + NT - 1) / NT;
  double v[kPer];
  int dst[kPer];
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int u = tid + NT * e, s = u / kSP, c = u - s * kSP;
    int t = -1;
    if (s < kSP) {
      if (s < nb2) t = kSP + s;
    } else if (s - kSP < nb2) {
      const int j = s - kSP, pj = S.piv[kSP + j];
      t = pj;
      if (pj < nb) t = -1;
      for (int j2 = 0; j2 < j; ++j2)
        if (S.piv[kSP + j2] == pj) t = -1;
    }
    dst[e] = -1;
    if (u < 2 * kSP * kSP && t >= 0) {
      const int src = swapped_source(t, S.piv, kSP, kSP + nb2);
      if (src != t) {
        v[e] = A[(size_t)(k0 + c) * m + k0 + src];
        dst[e] = t;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int u = tid + NT * e, c = u % kSP;
    if (dst[e] >= 0) A[(size_t)(k0 + c) * m + k0 + dst[e]] = v[e];
  }
}

// item = (leaf, c0, c1, mode): columns [c0, c1) of the leaf block.
// mode 0: left of the panel, the panel's swaps; 1: right of the panel, the
// panel's swaps then U12 = L11^{-1} A12; 3: U12 = L11^{-1} A12 only (columns
// right of an outer block, whose swaps were applied by lu_rowswap_kernel).
__global__ void __launch_bounds__(kUT) lu_strip_kernel(const int4* __restrict__ items, int k0,
                                                       const int2* __restrict__ leaf_rng,
                                                       const int64_t* __restrict__ blk_off,
                                                       double* __restrict__ lu,
                                                       const int* __restrict__ piv) {
  __shared__ double sL11[kBP][kBP + 1];
  __shared__ double sV[2 * kBP][kUC / 4];
  __shared__ int s_rows[2 * kBP], s_src[2 * kBP];
  __shared__ int s_idx[kPanelMaxM];
  __shared__ int s_nr;
  const int4 it = items[blockIdx.x];
  const int leaf = it.x, c0 = it.y, c1 = it.z, mode = it.w;
  const int2 lr = leaf_rng[leaf];
  const int m = 2 * lr.y;
  const int nb = min(kBP, m - k0);
  double* A = lu + blk_off[leaf];
  const int* ip = piv + 2 * lr.x;
  const int tid = threadIdx.x;
  const int ncol = c1 - c0;
  if (mode != 3) {
    // the panel's swaps replayed on the row indices k0..m-1, then the rows
    // whose content moved listed with the row their value comes from
    const int mr = m - k0;
    for (int i = tid; i < mr; i += kUT) s_idx[i] = k0 + i;
    if (tid == 0) s_nr = 0;
    __syncthreads();
    if (tid == 0)
      for (int j = 0; j < nb; ++j) {
        const int p = ip[k0 + j] - 1 - k0;
        const int t = s_idx[j];
        s_idx[j] = s_idx[p];
        s_idx[p] = t;
      }
    __syncthreads();
    for (int i = tid; i < mr; i += kUT)
      if (s_idx[i] != k0 + i) {
        const int q = atomicAdd(&s_nr, 1);  // at most 2 nb rows move
        s_rows[q] = k0 + i;
        s_src[q] = s_idx[i];
      }
    __syncthreads();
    const int nr = s_nr;
    for (int cs = 0; cs < ncol; cs += kUC / 4) {
      const int nc = min(kUC / 4, ncol - cs);
      for (int q = tid; q < nr * nc; q += kUT) {
        int row = q / nc, c = q - row * nc;
        sV[row][c] = A[(size_t)(c0 + cs + c) * m + s_src[row]];
      }
      __syncthreads();
      for (int q = tid; q < nr * nc; q += kUT) {
        int row = q / nc, c = q - row * nc;
        A[(size_t)(c0 + cs + c) * m + s_rows[row]] = sV[row][c];
      }
      __syncthreads();
    }
  }
  if (mode != 1 && mode != 3) return;
  for (int q = tid; q < nb * nb; q += kUT) {
    int c = q / nb, r = q - c * nb;
    sL11[r][c] = A[(size_t)(k0 + c) * m + k0 + r];
  }
  __syncthreads();
  if (tid < ncol) {  // U12 = L11^{-1} A12 (unit lower), one column per thread
    double* cc = A + (size_t)(c0 + tid) * m;
    double x[kBP];
#pragma unroll
    for (int r = 0; r < kBP; ++r) x[r] = (r < nb) ? cc[k0 + r] : 0.0;
#pragma unroll
    for (int r = 1; r < kBP; ++r) {
      double acc = x[r];
#pragma unroll
      for (int q = 0; q < kBP; ++q)
        if (q < r) acc = fma(-sL11[r][q], x[q], acc);
      x[r] = acc;
    }
#pragma unroll
    for (int r = 0; r < kBP; ++r)
      if (r < nb) cc[k0 + r] = x[r];
  }
}

// item = (leaf, r0, c0, ends): C[r0:r0+64, c0:c0+64] -= L[r0:, k0:k0+kd] U[k0:k0+kd, c0:]
// with kd = min(kdepth, m - k0) (32 inside a panel step, kOB for the update
// right of an outer block), staged 32 deep; rows are clipped at re and columns
// at ce, packed as ends = (re << 16) | ce (0: both m).  The C tile is read and
// written once per launch, so a 256-deep update moves an eighth of the bytes
// of eight 32-deep ones.
//
// The 32-deep slices of L and U are copied into shared memory with cp.async
// (16-byte chunks, zero-filled outside the tile), double-buffered: slice k+1
// is in flight while slice k is multiplied.  Every address is 16-byte
// aligned: blocks start at multiples of 4 doubles, m and all row and column
// offsets are even, and a slice's depth is even, so a chunk (two doubles) is
// either wholly inside the tile or wholly outside it.
constexpr int kUPitch = kBP + 2;  // U slice stored by column, 16-byte aligned rows
constexpr size_t kGemmSmem = sizeof(double) * 2 * (kBP * kGT + kGT * kUPitch);

__device__ __forceinline__ void cp_async16(double* dst, const double* src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src),
               "r"(valid ? 16 : 0));
}

__global__ void __launch_bounds__(kUT, 2) lu_gemm_kernel(const int4* __restrict__ items, int k0,
                                                         int kdepth,
                                                         const int2* __restrict__ leaf_rng,
                                                         const int64_t* __restrict__ blk_off,
                                                         double* __restrict__ lu) {
  extern __shared__ __align__(16) double gsm[];
  double* sLb = gsm;                      // [2][kBP][kGT]: L slice, k-major
  double* sUb = gsm + 2 * kBP * kGT;      // [2][kGT][kUPitch]: U slice, by column
  const int4 it = items[blockIdx.x];
  const int leaf = it.x, r0 = it.y, c0 = it.z;
  const int m = 2 * leaf_rng[leaf].y;
  const int re = it.w ? min(m, it.w >> 16) : m, ce = it.w ? min(m, it.w & 0xffff) : m;
  const int kd = min(kdepth, m - k0);
  double* A = lu + blk_off[leaf];
  const int tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
  // issue the copies of the slice starting at column k0 + kc into buffer buf
  auto load_slice = [&](int kc, int buf) {
    const int nbk = min(kBP, kd - kc), kb = k0 + kc;
    double* sL = sLb + buf * kBP * kGT;
    double* sU = sUb + buf * kGT * kUPitch;
#pragma unroll
    for (int e = 0; e < (kBP * kGT / 2) / kUT; ++e) {
      const int q = tid + kUT * e;
      const int k = q / (kGT / 2), rr = 2 * (q % (kGT / 2));
      const bool ok = k < nbk && r0 + rr < re;
      cp_async16(sL + k * kGT + rr, ok ? A + (size_t)(kb + k) * m + r0 + rr : A, ok);
    }
#pragma unroll
    for (int e = 0; e < (kGT * kBP / 2) / kUT; ++e) {
      const int q = tid + kUT * e;
      const int cc = q / (kBP / 2), kk = 2 * (q % (kBP / 2));
      const bool ok = kk < nbk && c0 + cc < ce;
      cp_async16(sU + cc * kUPitch + kk, ok ? A + (size_t)(c0 + cc) * m + kb + kk : A, ok);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  load_slice(0, 0);
  // C values first (independent of the tiles)
  double cv[4][4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int c = c0 + tc + 16 * b;
    const double* cc = A + (size_t)c * m;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int r = r0 + tr + 16 * a;
      cv[a][b] = (c < ce && r < re) ? cc[r] : 0.0;
    }
  }
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
  for (int kc = 0, buf = 0; kc < kd; kc += kBP, buf ^= 1) {
    if (kc + kBP < kd) {
      load_slice(kc + kBP, buf ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::);
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::);
    }
    __syncthreads();
    const double* sL = sLb + buf * kBP * kGT;
    const double* sU = sUb + buf * kGT * kUPitch;
#pragma unroll 8
    for (int k = 0; k < kBP; ++k) {
      double lv[4], uv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) lv[a] = sL[k * kGT + tr + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) uv[b] = sU[(tc + 16 * b) * kUPitch + k];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fma(lv[a], uv[b], acc[a][b]);
    }
    __syncthreads();  // buffer buf is refilled two slices on
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int c = c0 + tc + 16 * b;
    if (c >= ce) continue;
    double* cc = A + (size_t)c * m;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int r = r0 + tr + 16 * a;
      if (r < re) cc[r] = cv[a][b] - acc[a][b];
    }
  }
}

// Row interchanges of an outer block (pivots K0 .. K0+nb-1, in order) as one
// gather: per leaf (one CTA), the swaps are replayed on an index array of the
// rows K0.. in shared memory, then the rows whose content moved are listed
// with the row their value comes from (map row of the leaf: 2 kOB rows, 2 kOB
// sources, count; stride 4 kOB + 1 ints).
__global__ void __launch_bounds__(256) lu_swapmap_kernel(const int* __restrict__ leaves, int K0,
                                                         const int2* __restrict__ leaf_rng,
                                                         const int* __restrict__ piv,
                                                         int* __restrict__ map) {
  __shared__ int idx[kPanelMaxM];
  __shared__ int cnt;
  const int leaf = leaves[blockIdx.x];
  const int2 lr = leaf_rng[leaf];
  const int m = 2 * lr.y, nb = min(kOB, m - K0), mr = m - K0;
  const int* ip = piv + 2 * lr.x;
  int* rows = map + (size_t)blockIdx.x * (4 * kOB + 1);
  int* src = rows + 2 * kOB;
  for (int i = threadIdx.x; i < mr; i += blockDim.x) idx[i] = K0 + i;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int j = 0; j < nb; ++j) {
      const int p = ip[K0 + j] - 1 - K0;
      const int t = idx[j];
      idx[j] = idx[p];
      idx[p] = t;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < mr; i += blockDim.x)
    if (idx[i] != K0 + i) {
      const int q = atomicAdd(&cnt, 1);  // at most 2 nb rows move
      rows[q] = K0 + i;
      src[q] = idx[i];
    }
  __syncthreads();
  if (threadIdx.x == 0) rows[4 * kOB] = cnt;
}

// item = (slot, c0, c1, leaf): the outer block's row interchanges on columns
// [c0, c1), through the map of lu_swapmap_kernel (slot = the leaf's map row)
constexpr int kRC = 8;  // columns per pass
__global__ void __launch_bounds__(kUT) lu_rowswap_kernel(const int4* __restrict__ items,
                                                         const int2* __restrict__ leaf_rng,
                                                         const int64_t* __restrict__ blk_off,
                                                         const int* __restrict__ map,
                                                         double* __restrict__ lu) {
  __shared__ double sV[2 * kOB][kRC];
  const int4 it = items[blockIdx.x];
  const int* rows = map + (size_t)it.x * (4 * kOB + 1);
  const int* src = rows + 2 * kOB;
  const int nr = rows[4 * kOB];
  const int m = 2 * leaf_rng[it.w].y;
  double* A = lu + blk_off[it.w];
  for (int cs = it.y; cs < it.z; cs += kRC) {
    const int nc = min(kRC, it.z - cs);
    for (int q = threadIdx.x; q < nr * nc; q += kUT) {
      const int row = q / nc, c = q - row * nc;
      sV[row][c] = A[(size_t)(cs + c) * m + src[row]];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nr * nc; q += kUT) {
      const int row = q / nc, c = q - row * nc;
      A[(size_t)(cs + c) * m + rows[row]] = sV[row][c];
    }
    __syncthreads();
  }
}

// After the factorisation, per leaf: the row permutation of all its pivots
// (DLASWP applied to the index vector, so an apply gathers in one parallel
// step) and the inverses of the 32 x 32 diagonal blocks of L (unit lower) and
// U (upper), so that each step of the blocked substitutions is a small GEMV
// instead of a 32-step serial recurrence.
constexpr int kDB = 32;

__global__ void lu_perm_kernel(const int2* __restrict__ leaf_rng, const int* __restrict__ piv,
                               int nleaf, int* __restrict__ perm) {
  int leaf = blockIdx.x * blockDim.x + threadIdx.x;
  if (leaf >= nleaf) return;
  int2 lr = leaf_rng[leaf];
  int m = 2 * lr.y;
  const int* ip = piv + 2 * lr.x;
  int* pm = perm + 2 * lr.x;
  for (int i = 0; i < m; ++i) pm[i] = i;
  for (int k = 0; k < m; ++k) {
    int p = ip[k] - 1;
    if (p != k) {
      int t = pm[k];
      pm[k] = pm[p];
      pm[p] = t;
    }
  }
}

// one warp per (leaf, diagonal block): lane j computes column j of L^{-1} and
// U^{-1} of the block (identity padding past the end of the matrix)
__global__ void lu_diaginv_kernel(const int2* __restrict__ blocks,  // (leaf, k0)
                                  const int2* __restrict__ leaf_rng,
                                  const int64_t* __restrict__ blk_off,
                                  const int64_t* __restrict__ dinv_off,
                                  const double* __restrict__ lu, double* __restrict__ dinv,
                                  int* __restrict__ info) {
  __shared__ double D[4][kDB][kDB + 1];
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int2 bk = blocks[blockIdx.x * 4 + w];
  if (bk.x < 0) return;
  int2 lr = leaf_rng[bk.x];
  int m = 2 * lr.y, k0 = bk.y, nb = min(kDB, m - k0);
  const double* A = lu + blk_off[bk.x];
  for (int c = 0; c < kDB; ++c)
    D[w][lane][c] = (c < nb && lane < nb) ? A[(size_t)(k0 + c) * m + k0 + lane]
                                          : (c == lane ? 1.0 : 0.0);
  __syncwarp();
  // a NaN or Inf pivot (coincident faces give a non-finite kernel value) is
  // recorded as -(its 1-based row); DGETRF's exact-zero info takes precedence
  if (lane < nb && !isfinite(D[w][lane][lane])) atomicCAS(&info[bk.x], 0, -(k0 + lane + 1));
  double* Li = dinv + dinv_off[bk.x] + (size_t)(k0 / kDB) * 2 * kDB * kDB;
  double* Ui = Li + kDB * kDB;
  // L^{-1} e_j (unit lower)
  double x[kDB];
#pragma unroll
  for (int i = 0; i < kDB; ++i) {
    double v = (i == lane) ? 1.0 : 0.0;
#pragma unroll
    for (int q = 0; q < kDB; ++q)
      if (q < i) v = fma(-D[w][i][q], x[q], v);
    x[i] = v;
  }
#pragma unroll
  for (int i = 0; i < kDB; ++i) Li[(size_t)lane * kDB + i] = x[i];  // column lane
  // U^{-1} e_j (upper, non-unit)
#pragma unroll
  for (int i = kDB - 1; i >= 0; --i) {
    double v = (i == lane) ? 1.0 : 0.0;
#pragma unroll
    for (int q = 0; q < kDB; ++q)
      if (q > i) v = fma(-D[w][i][q], x[q], v);
    x[i] = v / D[w][i][i];
  }
#pragma unroll
  for (int i = 0; i < kDB; ++i) Ui[(size_t)lane * kDB + i] = x[i];
}

// Forward/back substitution with the factored block (DGETRS 'N'), one CTA per
// leaf: gather through the pivot permutation, then L and U in 32-row steps.
// Step t needs sum_u T(t,u) y_u over the earlier steps' 32 x 32 tiles T and
// the precomputed inverse of its diagonal block, y_t = Dinv (r_t - sum).
//
// The tiles of both sweeps form one sequence, known from the start, in the
// order they are needed, so eight warps copy them into a ring of RING tiles by
// cp.async well ahead of their use and the loads wait for nothing but the ring;
// a thread copies the 16-byte chunks (two rows of two columns) that it
// multiplies itself, so a tile costs no barrier.  Per step, T(t,t-1) y_{t-1}
// is the only product that waits for the step before; then, while the ninth
// warp forms y_t, the others already sum step t+1's tiles with u < t.  Two
// barriers per step.
//
// Bound by the chain of steps (two barriers, the sums across warps and a 32-deep
// dot product each, 0.6 us) and, for blocks of order ~1,000, by one SM's rate of
// taking tiles.  The form before this one updated all rows below (above) with
// each y, so every step's panel loads were issued after its barrier and waited
// for memory.  Per apply: 2,544 unknowns in blocks of ~320 41 -> 30 us;
// 121,352 unknowns (590 MB of factors) 171 -> 156 us; 186,260 unknowns (800 MB)
// 176 -> 168 us with L2 flushed, in blocks of 200 79 -> 53 us, of 60 92 -> 70 us;
// 807,640 unknowns (1,970 MB) 395 -> 361 us.
//
// Blocks of order > 512: two groups of eight warps, each with a ring of nine
// tiles (one group: 210 us where two take 182), which shared memory holds up to
// order 6,912.  The others: one group and five tiles, so that three CTAs share
// an SM (two CTAs with six tiles: 383 instead of 375 us for 807,640 unknowns in
// blocks of ~300).  Taking two or three tiles per wait keeps fewer in flight: 607
// and 643 instead of 573 us at order 2,464 with L2 flushed (623 before), 170 and
// 174 instead of 166 us for 800 MB.  Blocks whose factors stay in L2, and lone ones
// of an odd number of faces: solve_rows_kernel.
constexpr int kTile = kDB * kDB, kDRing = 3, kRingBig = 9, kRingSmall = 5;
constexpr int kRingHuge = 6, kSolveHuge = 6912;  // blocks above this order
constexpr int kMaxSolveLeaf = 5760;  // faces

// threads and shared memory of solve_kernel<G, RING> for a block of the given order
constexpr int solve_threads(int G) { return 256 * G + 32; }
constexpr size_t solve_bytes(int G, int RING, int order) {
  return sizeof(double) * ((size_t)(order + kDB - 1) / kDB * kDB + (8 * G + 1) * kDB +
                           kDRing * kTile + G * RING * kTile);
}

template <int G, int RING>
__global__ void __launch_bounds__(solve_threads(G), (G == 1 ? 3 : 1)) solve_kernel(
    const int2* __restrict__ leaf_rng, const int64_t* __restrict__ blk_off,
    const int64_t* __restrict__ dinv_off, const int* __restrict__ leaf_list,
    const double* __restrict__ lu, const double* __restrict__ dinv,
    const int* __restrict__ perm, int N, const double* __restrict__ r,
    double* __restrict__ z) {
  extern __shared__ __align__(16) double sm[];
  const int leaf = leaf_list[blockIdx.x];
  const int2 lr = leaf_rng[leaf];
  const int n = lr.y, m = 2 * n, ib = lr.x;
  const int nblk = (m + kDB - 1) / kDB;
  double* vec = sm;                       // r, then y, then x (zero past m)
  double* part = vec + kDB * nblk;        // [8 G][32] the warps' sums
  double* sv = part + 8 * G * kDB;            // [32] the step's right-hand side
  double* dbuf = sv + kDB;                // [kDRing] inverse diagonal blocks
  double* ring = dbuf + kDRing * kTile;   // [G][RING] tiles, by column
  const double* A = lu + blk_off[leaf];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int* pm = perm + 2 * ib;
  auto copy16 = [](double* dst, const double* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
  };
  auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
  // block of sweep `back`'s step t
  auto block = [&](int back, int t) { return back ? nblk - 1 - t : t; };
  if (warp == 8 * G) {
    // the chain: inverse diagonal blocks kDRing - 1 steps ahead
    const double* Di = dinv + dinv_off[leaf];
    auto stage = [&](int q) {  // step q of both sweeps
      if (q < 2 * nblk) {
        const int back = q >= nblk, b = block(back, back ? q - nblk : q);
        const double* src = Di + (size_t)b * 2 * kTile + (back ? kTile : 0);
        double* dst = dbuf + (q % kDRing) * kTile;
#pragma unroll
        for (int e = 2 * lane; e < kTile; e += 64) copy16(dst + e, src + e, true);
      }
      commit();
    };
    for (int q = 0; q < kDRing - 1; ++q) stage(q);
    __syncthreads();  // vec
    for (int q = 0; q < 2 * nblk; ++q) {
      const int back = q >= nblk, b = block(back, back ? q - nblk : q);
      stage(q + kDRing - 1);
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kDRing - 1) : "memory");
      __syncthreads();  // the warps' sums
      double p[4] = {};
#pragma unroll
      for (int w = 0; w < 8 * G; ++w) p[w & 3] += part[w * kDB + lane];
      sv[lane] = vec[kDB * b + lane] - ((p[0] + p[1]) + (p[2] + p[3]));
      __syncwarp();
      const double* D = dbuf + (q % kDRing) * kTile + lane;
      const double2* s2 = reinterpret_cast<const double2*>(sv);
      double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
#pragma unroll
      for (int k = 0; k < kDB; k += 4) {
        const double2 a = s2[k / 2], c = s2[k / 2 + 1];
        v0 = fma(D[k * kDB], a.x, v0);
        v1 = fma(D[(k + 1) * kDB], a.y, v1);
        v2 = fma(D[(k + 2) * kDB], c.x, v2);
        v3 = fma(D[(k + 3) * kDB], c.y, v3);
      }
      vec[kDB * b + lane] = (v0 + v1) + (v2 + v3);
      __syncthreads();  // y_t
    }
  } else {
    // group g takes the tiles of the source steps u = g modulo G; this thread's
    // rows and columns of a tile:
    const int g = warp >> 3, rp = 2 * (tid & 15), cp = 2 * ((tid >> 4) & 15);
    double* const mine = ring + g * RING * kTile + cp * kDB + rp;
    double* const last = mine + (RING - 1) * kTile;
    // the tile to copy next: sweep, step, tiles left in the step, offset in A, column
    int ps = g + 1 < nblk ? 0 : 2, pt = g + 1, left = 1, off = 0, pj = 0;
    bool rows = false;
    const unsigned first = (unsigned)__cvta_generic_to_shared(mine);
    unsigned dst = first;
    auto strip = [&] {  // first tile of step pt
      const int i = kDB * block(ps, pt) + rp;
      pj = kDB * block(ps, g) + cp;
      rows = i < m;
      off = pj * m + i;
      left = (pt - g + G - 1) / G;
    };
    if (ps < 2) strip();
    auto issue = [&] {
      if (ps < 2) {
        const bool ok = rows && pj < m;  // m, the row and the column are even
        const double* src = A + (ok ? off : 0);
        const int size = ok ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                     "cp.async.cg.shared.global [%0 + %4], [%3], 16, %2;\n" ::"r"(dst),
                     "l"(src), "r"(size), "l"(src + (ok ? m : 0)), "n"(kDB * sizeof(double))
                     : "memory");
        const int d = ps ? -G * kDB : G * kDB;
        off += d * m;
        pj += d;
        if (--left == 0) {
          if (++pt == nblk) {
            pt = g + 1;
            ++ps;
          }
          if (ps < 2) strip();
        }
      }
      dst = dst == first + (RING - 1) * kTile * (unsigned)sizeof(double)
                ? first
                : dst + kTile * (unsigned)sizeof(double);
      commit();
    };
#pragma unroll 1
    for (int q = 0; q < RING - 1; ++q) issue();
    for (int i = tid; i < kDB * nblk; i += 256 * G) {
      double v = 0.0;
      if (i < m) {
        const int k = pm[i];
        v = (k < n) ? r[ib + k] : r[N + ib + k - n];
      }
      vec[i] = v;
    }
    double a00 = 0.0, a10 = 0.0, a01 = 0.0, a11 = 0.0;  // rows rp, rp + 1 by columns cp, cp + 1
    const double* t = mine;
    auto mul = [&](const double* v) {  // the ring's next tile times y
      const double2 x = *reinterpret_cast<const double2*>(t);
      const double2 y = *reinterpret_cast<const double2*>(t + kDB);
      const double2 w = *reinterpret_cast<const double2*>(v);
      a00 = fma(x.x, w.x, a00);
      a10 = fma(x.y, w.x, a10);
      a01 = fma(y.x, w.y, a01);
      a11 = fma(y.y, w.y, a11);
      t = t == last ? mine : t + kTile;
    };
    __syncthreads();  // vec
    for (int back = 0; back < 2; ++back) {
      const int d = back ? -G * kDB : G * kDB;  // from a source step of the group to its next
      const double* v0 = vec + kDB * block(back, g) + cp;
      for (int q = 0; q < nblk; ++q) {
        const bool prev = q > 0 && (q - 1) % G == g;
        if (prev) {
          asm volatile("cp.async.wait_group %0;\n" ::"n"(RING - 2) : "memory");
          mul(vec + kDB * block(back, q - 1) + cp);
        }
        double s0 = a00 + a01, s1 = a10 + a11;
        s0 += __shfl_xor_sync(0xffffffffu, s0, 16);
        s1 += __shfl_xor_sync(0xffffffffu, s1, 16);
        if (lane < 16) *reinterpret_cast<double2*>(part + warp * kDB + rp) = make_double2(s0, s1);
        a00 = a10 = a01 = a11 = 0.0;
        __syncthreads();  // the warps' sums
        if (prev) issue();
        if (q + 1 < nblk) {
          const double* v = v0;
#pragma unroll 1
          for (int u = g; u < q; u += G, v += d) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(RING - 2) : "memory");
            mul(v);
            issue();  // into the slot of the tile before this one
          }
        }
        __syncthreads();  // y_t
      }
    }
  }
  for (int i = tid; i < n; i += solve_threads(G)) {
    z[ib + i] = vec[i];
    z[N + ib + i] = vec[n + i];
  }
}

// The same substitution with the factors read where they are used: per step the first
// warp forms y_t = Dinv r_t, and 512 threads update the rows below (above) with the
// step's 32 columns, each thread a row, the first row's values loaded while y_t is
// formed.  Every step's loads wait for its barrier, but a 32 x 32 tile costs a fifth
// of the streamed form's instructions, which bound that form once the factors come
// from L2, and its loads are whole rows of columns, where the streamed 16-byte
// copies straddle sectors in the columns of an odd number of faces.
//
// Taken where the factors of all leaves stay in L2 even beside two more handles at
// work (kRowBytes), us per apply of this form and the streamed one, one handle and
// three in turn: 10 MB in blocks of up to 558 unknowns 41.4, 44.5 and 14.8, 15.5;
// 20 MB, one block of 978, 97, 106 and 35.4, 36.3; not at 25 MB, blocks up to 754,
// 66, 69 and 31, 25; 39 MB, up to 844, 76, 78 and 37, 29; 96 MB, up to 664, 75, 55
// and 36, 28.  And for a lone block (there is nothing beside it to fill an SM) up to
// kLoneBytes, order 2,000 302, 333 and 121, 113, 2,464 427, 478 and 189, 162, or of an
// odd number of faces up to kLoneOrder: order 2,502 476, 587 and 206, 199; 3,502
// 991, 1,111 and 372, 372; 7,002 4,040, 4,287 and 1,339, 1,428; beyond, 8,002 5,774,
// 5,590; an even number, 2,900 680, 661 and 266, 222.
constexpr int kRowThreads = 512;
constexpr int64_t kRowBytes = 20 << 20, kLoneBytes = 56 << 20;
constexpr int kLoneOrder = 7500;
constexpr size_t row_bytes(int order) {
  return sizeof(double) * (2 * (size_t)order + kDB + 2 * kTile);
}

__global__ void __launch_bounds__(kRowThreads, 1) solve_rows_kernel(
    const int2* __restrict__ leaf_rng, const int64_t* __restrict__ blk_off,
    const int64_t* __restrict__ dinv_off, const int* __restrict__ leaf_list,
    const double* __restrict__ lu, const double* __restrict__ dinv,
    const int* __restrict__ perm, int N, const double* __restrict__ r,
    double* __restrict__ z) {
  extern __shared__ __align__(16) double sm[];
  int leaf = leaf_list[blockIdx.x];
  int2 lr = leaf_rng[leaf];
  const int n = lr.y, m = 2 * n, ib = lr.x;
  double* xs = sm;             // forward sweep: running; backward: results
  double* fin = sm + m;        // forward sweep: results; backward: running
  double* ys = sm + 2 * m;     // [32] the step's y
  const double* A = lu + blk_off[leaf];
  const double* Di = dinv + dinv_off[leaf];
  const int* pm = perm + 2 * ib;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < m; i += kRowThreads) {
    int src = pm[i];
    xs[i] = (src < n) ? r[ib + src] : r[N + ib + src - n];
  }
  // the inverse diagonal block of sweep step t (L blocks 0..nblk-1, then U
  // blocks nblk-1..0), staged into shared memory one step ahead by cp.async
  const int nblk = (m + kDB - 1) / kDB;
  double* dbuf = ys + kDB;  // [2][kDB * kDB]
  auto stage = [&](int t, int buf) {
    if (t >= 2 * nblk) return;
    const int b = t < nblk ? t : 2 * nblk - 1 - t;
    const double* src = Di + (size_t)b * 2 * kDB * kDB + (t < nblk ? 0 : kDB * kDB);
    for (int e = 2 * tid; e < kDB * kDB; e += 2 * kRowThreads) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(dbuf + buf * kDB * kDB + e);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + e));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  // step t: y = Dinv * run[k0 .. k0+nb), res[k0 ..] = y, run[i] -= A[i, k0 ..
  // k0+nb) y for the rows [i0, i1); the next step's block is copied while the
  // rows are updated.  Four partial sums per dot product keep the dependent
  // FMA chains 8 deep.
  // y = Dinv * run[k0 .. k0+nb) for lane `lane`, four partial sums
  auto diag = [&](int t, int k0, int nb, const double* run) {
    const double* Dblk = dbuf + (t & 1) * kDB * kDB;
    double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
    if (nb == kDB) {  // run + k0 is 16-byte aligned: paired loads
      const double2* r2 = reinterpret_cast<const double2*>(run + k0);
#pragma unroll
      for (int q = 0; q < kDB; q += 4) {
        const double2 ra = r2[q / 2], rb = r2[q / 2 + 1];
        v0 = fma(Dblk[q * kDB + lane], ra.x, v0);
        v1 = fma(Dblk[(q + 1) * kDB + lane], ra.y, v1);
        v2 = fma(Dblk[(q + 2) * kDB + lane], rb.x, v2);
        v3 = fma(Dblk[(q + 3) * kDB + lane], rb.y, v3);
      }
    } else {
      for (int q = 0; q < nb; ++q) v0 = fma(Dblk[q * kDB + lane], run[k0 + q], v0);
    }
    return (v0 + v1) + (v2 + v3);
  };
  // run[i] -= A[i, k0 .. k0+nb) y for row i, tq preloaded when `have`
  auto row = [&](int k0, int nb, int i, const double* y, double (&tq)[kDB], bool have,
                 double* run) {
    const double* a = A + (size_t)k0 * m + i;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    if (nb == kDB) {
      if (!have) {
#pragma unroll
        for (int q = 0; q < kDB; ++q) tq[q] = a[(size_t)q * m];
      }
      const double2* y2 = reinterpret_cast<const double2*>(y);
#pragma unroll
      for (int q = 0; q < kDB; q += 4) {
        const double2 ya = y2[q / 2], yb = y2[q / 2 + 1];
        s0 = fma(tq[q], ya.x, s0);
        s1 = fma(tq[q + 1], ya.y, s1);
        s2 = fma(tq[q + 2], yb.x, s2);
        s3 = fma(tq[q + 3], yb.y, s3);
      }
    } else {
      for (int q = 0; q < nb; ++q) s0 = fma(a[(size_t)q * m], y[q], s0);
    }
    run[i] -= (s0 + s1) + (s2 + s3);
  };
  auto step = [&](int t, int k0, int nb, double* run, double* res, int i0, int i1) {
    double tq[kDB];
    // warp 0 forms y and shares it through shared memory (one more barrier,
    // against 16 warps each reading the 8 KB block); the first row's panel
    // values are loaded meanwhile
    const int ifirst = i0 + tid;
    const bool pre = ifirst < i1 && nb == kDB;
    if (pre) {
      const double* a = A + (size_t)k0 * m + ifirst;
#pragma unroll
      for (int q = 0; q < kDB; ++q) tq[q] = a[(size_t)q * m];
    }
    if (warp == 0) {
      const double v = diag(t, k0, nb, run);
      ys[lane] = v;
      if (lane < nb) res[k0 + lane] = v;
    }
    stage(t + 1, (t + 1) & 1);
    __syncthreads();
    for (int i = ifirst; i < i1; i += kRowThreads) row(k0, nb, i, ys, tq, pre && i == ifirst, run);
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
  };
  stage(0, 0);
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  // L y = P r: running values in xs, y in fin
  for (int k0 = 0, t = 0; k0 < m; k0 += kDB, ++t) {
    const int nb = min(kDB, m - k0);
    step(t, k0, nb, xs, fin, k0 + nb, m);
  }
  // U x = y: running values in fin, x in xs
  for (int b = nblk - 1, t = nblk; b >= 0; --b, ++t) {
    const int k0 = b * kDB;
    const int nb = min(kDB, m - k0);
    step(t, k0, nb, fin, xs, 0, k0);
  }
  for (int i = tid; i < n; i += kRowThreads) {
    z[ib + i] = xs[i];
    z[N + ib + i] = xs[n + i];
  }
}

// ---------------------------------------------------------------------------
// Unpivoted blocked LU with a certificate of partial pivoting.
//
// DGETRF2 swaps rows only where a column holds an entry larger in magnitude
// than its diagonal after elimination (IDAMAX, first index on ties).  The leaf
// blocks of a well-resolved surface are strongly diagonal (the 2n x 2n blocks
// of the benchmark molecule have condition numbers near 100 and no row
// interchange at all), so the factorisation runs first without pivot
// searches, right-looking in outer blocks of 128 columns, three launches each
// over all leaves of a group:
//   lu_np_block_kernel   the 128 x 128 diagonal block of every leaf, one CTA
//                        each, in two 64-column steps, with the inverses of
//                        the 64 x 64 diagonal blocks' L and U (and their
//                        32 x 32 diagonal blocks for the applies);
//   lu_np_border_kernel  the block's L21 = A21 U11^{-1} by 64-row chunks and
//                        U12 = L11^{-1} A12 by 64-column chunks: each chunk's
//                        two 64-deep steps depend on no other chunk, so one
//                        CTA takes them all from shared memory;
//   lu_gemm2_kernel      A22 -= L21 U12, 128 deep.
// Every multiplier l is checked: |l| <= 1 - 2^-20 for all of them certifies
// that partial pivoting (on these values or on the reference's, which differ
// by rounding only) keeps the diagonal row at every column, so the factors
// are DGETRF's.  A leaf whose certificate fails anywhere (a larger entry, a
// near tie, a zero or non-finite pivot) is re-assembled and factored again by
// the pivoted kernels above.
constexpr int kNP = 64;    // step width
constexpr int kNPT = 256;  // threads of the block kernel
constexpr int kOB2 = 128;  // outer block
constexpr int kPP = kNP + 4;  // pitch of a staged 64-double column
constexpr int kNB2 = kNP * kPP;  // a staged 64 x 64 block
constexpr double kNoPivBound = 1.0 - 1.0 / 1048576.0;

// FP64 tensor-core product of 8 x 8 x 4 (tcgen05 has no FP64 kind; this one runs
// at the FP64 pipe's full rate, 37.05 TFLOP/s measured against 36.7 of a DFMA
// loop, with an eighth of the instructions and shared loads).  Lane l holds
// A[l / 4][l % 4], B[l % 4][l / 4] and C[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// acc += A B for a warp's (8 MT) x (8 NT) tile over KD (a multiple of 4): A
// k-major (row r, depth k at A[k * AP + r]), B by column (depth k, column c at
// B[c * BP + k]).  A pitch of 4 modulo 16 doubles puts the 16 words of a
// half-warp's fragment load on 16 different bank pairs.
template <int MT, int NT, int AP, int BP, int KD>
__device__ __forceinline__ void dmma_tile(double (&acc)[MT][NT][2], const double* A,
                                          const double* B) {
  static_assert(AP % 16 == 4 && BP % 16 == 4, "fragment loads on different banks");
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const double* a = A + t * AP + g;
  const double* b = B + g * BP + t;
#pragma unroll
  for (int k = 0; k < KD; k += 4) {
    double av[MT], bv[NT];
#pragma unroll
    for (int i = 0; i < MT; ++i) av[i] = a[k * AP + 8 * i];
#pragma unroll
    for (int i = 0; i < NT; ++i) bv[i] = b[8 * i * BP + k];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int q = 0; q < NT; ++q) dmma884(acc[i][q], av[i], bv[q]);
  }
}

// The same over the first kd (16, 32, 48 or 64) of 64: for a triangular operand,
// whose later part is zero for this tile (border of a 128-column block, 31 leaves of
// order ~1400: 88.7 -> 77.6 us for the columns, 86.6 -> 82.5 us for the rows).
template <int MT, int NT, int AP, int BP>
__device__ __forceinline__ void dmma_tile_part(double (&acc)[MT][NT][2], const double* A,
                                               const double* B, int kd) {
#pragma unroll 1
  for (int k = 0; k < kd; k += 16)
    dmma_tile<MT, NT, AP, BP, 16>(acc, A + k * AP, B + k);
}

// Copies a block of 64 columns of 64 doubles (leading dimension ld, 16-byte
// aligned columns) into shared memory at pitch kPP, zeros outside nr x nc (nr
// even); the caller commits and waits.  NT: threads of the CTA.
template <int NT>
__device__ __forceinline__ void stage64(double* dst, const double* src, int ld, int nr, int nc) {
#pragma unroll
  for (int e = 0; e < kNP * kNP / 2 / NT; ++e) {
    const int q = (int)threadIdx.x + NT * e, c = q >> 5, r = 2 * (q & 31);
    const bool ok = c < nc && r < nr;
    cp_async16(dst + c * kPP + r, ok ? src + (size_t)c * ld + r : src, ok);
  }
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// f(r, c, entry) over the lane's entries of a warp's (8 MT) x (8 NT) tile
template <int MT, int NT, typename F>
__device__ __forceinline__ void tile_each(double (&acc)[MT][NT][2], F&& f) {
  const int r = (int)(threadIdx.x & 31) >> 2, c = 2 * ((int)threadIdx.x & 3);
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int q = 0; q < NT; ++q)
#pragma unroll
      for (int b = 0; b < 2; ++b) f(r + 8 * i, c + 8 * q + b, acc[i][q][b]);
}

// 1/x to about an ulp for x from the smallest normal to kRcpMax: one third-order
// Householder step y (1 + e + e^2), e = 1 - x y, from the hardware's approximation
// (relative error 2^-20); a chain of four operations after it, half the latency
// of a division.  Above 2^1022 the reciprocal is subnormal and the approximation
// gives 0.
constexpr double kRcpMax = 0x1p1021;
__device__ __forceinline__ double fast_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// The CTA (256 threads, one element each): the 16 x 16 block at A (shared,
// column-major, pitch kPP; rows and columns from d on are zero) factored in
// place without interchanges (DGETRF2's scaling: multipliers times the pivot's
// reciprocal); rcp receives the reciprocals of the pivots (0 from d on).  True
// in threads whose entry fails the certificate; a pivot that is zero, subnormal
// (where DGETRF2 divides instead), above kRcpMax or not finite fails it too, and
// the leaf goes to the pivoted kernels, which follow DGETRF2 there.  Step t reads row and
// column t and writes only entries right of and below them, so one barrier a
// step is enough.  One warp with eight entries a lane took 475 cycles a step
// (its own 110 instructions), one entry a thread takes a third of that.
__device__ __forceinline__ bool lu_diag16(double* A, int d, double* rcp) {
  const int r = threadIdx.x & 15, c = threadIdx.x >> 4;
  double a = A[c * kPP + r];
#pragma unroll 1
  for (int t = 0; t < d; ++t) {
    const double rp = fast_rcp(A[t * kPP + t]);
    const double l = A[t * kPP + r] * rp, u = A[c * kPP + t];
    if (r > t) {
      if (c > t) {
        a = fma(-l, u, a);
        A[c * kPP + r] = a;
      } else if (c == t) {
        a = l;
      }
    }
    if (r == t && c == t) rcp[t] = rp;
    __syncthreads();
  }
  bool bad = false;
  if (r > c) {
    A[c * kPP + r] = a;
    bad = !(fabs(a) <= kNoPivBound);
  } else if (r == c) {
    if (r < d)
      bad = !(fabs(a) >= 2.2250738585072014e-308 && fabs(a) <= kRcpMax);
    else
      rcp[r] = 0.0;
  }
  return bad;
}

// One warp: li and ui (zero on entry) receive the inverses of the factored 16 x
// 16 block at A, zero from d on.  Half h = 0 of the warp: column r of L^{-1} by
// forward substitution; h = 1: column r of U^{-1} by backward substitution, the
// same loop on reversed indices.
__device__ __forceinline__ void lu_inv16(const double* A, int d, const double* rcp, double* li,
                                         double* ui) {
  const int lane = threadIdx.x & 31, r = lane & 15, h = lane >> 4;
  const double* M = h == 0 ? A : A + 15 * kPP + 15;
  const int sg = h == 0 ? 1 : -1, c = h == 0 ? r : 15 - r;
  double x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = i == c && r < d ? 1.0 : 0.0;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    if (h == 1) x[q] *= rcp[15 - q];
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i > q) x[i] = fma(-M[sg * (q * kPP + i)], x[q], x[i]);
  }
  double* out = (h == 0 ? li : ui) + r * kPP;
#pragma unroll
  for (int i = 0; i < 16; ++i) out[h == 0 ? i : 15 - i] = x[i];
}

// The d x d (d <= 64) diagonal block at D (column-major, leading dimension m)
// factored in place; li and ui (shared, pitch kPP) receive L^{-1} (unit lower)
// and U^{-1}, column-major with zeros outside the triangle and from d on (d <= 32:
// their first 32 columns only); S (null: not wanted, which it is only beside a
// border and so with d = 64) the same at pitch 64; Di their 32 x 32 diagonal blocks
// (identity padded, the layout lu_diaginv_kernel writes).  fb: shared scratch of one staged block.
// Every thread of the CTA; true if the certificate failed in an entry of this
// thread.  Right-looking in four 16-column steps: the CTA factors the 16 x 16
// block, a lane each substitutes a row of L or a column of U, and the update
// is 16 x 16 x 16 tensor-core products, one warp each.  Then the inverses of the
// four 16 x 16 blocks, one warp each, and from them by doubling those of 32 and
// 64.  A loop over 64 columns with
// one CTA barrier each, forming both inverses on the way, took 600 cycles a
// column.  What a block of up to 32 columns, or one without a border, does not need is
// left out: 19,000 leaves of 10 faces 821 -> 517 us.
__device__ bool lu_diag64(double* D, int m, int d, double* li, double* ui, double* fb,
                          double* s_rcp, double* S, double* Di) {
  const int tid = threadIdx.x, warp = tid >> 5;
  constexpr int B = 16 * (kPP + 1);  // from one 16 x 16 diagonal block to the next
  constexpr int C = 16 * kPP, NB = 4;
  stage64<kNPT>(fb, D, m, d, d);
  cp_async_commit();
  // a block of up to 32 columns is in the first 32 of each buffer
  for (int e = tid; e < (d <= kDB ? kNB2 / 2 : kNB2); e += kNPT) li[e] = ui[e] = 0.0;
  cp_async_wait<0>();
  __syncthreads();
  bool bad = false;
  auto put = [](double* dst, double (&acc)[2][2][2], double s) {
    tile_each(acc, [&](int r, int c, double v) { dst[c * kPP + r] = s * v; });
  };
  for (int j = 0; 16 * j < d; ++j) {
    double* a = fb + j * B;
    double* rcp = s_rcp + 16 * j;
    bad |= lu_diag16(a, min(16, d - 16 * j), rcp);
    __syncthreads();
    // warps 0 and 1: row 16 + lane of L below the block; 2 and 3: column of U
    // right of it
    const int rem = NB - 1 - j, x0 = tid & 63;
    if (tid < 128 && x0 < 16 * rem) {
      double x[16];
      if (tid < 64) {
        double* p = a + 16 + x0;
#pragma unroll
        for (int q = 0; q < 16; ++q) x[q] = p[q * kPP];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          x[q] *= rcp[q];
          if (!(fabs(x[q]) <= kNoPivBound)) bad = true;
#pragma unroll
          for (int c = q + 1; c < 16; ++c) x[c] = fma(-x[q], a[c * kPP + q], x[c]);
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) p[q * kPP] = x[q];
      } else {
        double* p = a + (16 + x0) * kPP;
#pragma unroll
        for (int q = 0; q < 16; ++q) x[q] = p[q];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
#pragma unroll
          for (int i = q + 1; i < 16; ++i) x[i] = fma(-a[q * kPP + i], x[q], x[i]);
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) p[q] = x[q];
      }
    }
    __syncthreads();
    for (int w = warp; w < rem * rem; w += kNPT / 32) {
      const int i = w % rem + 1, k = w / rem + 1;
      double* t = a + 16 * i + k * C;
      double acc[2][2][2];
      tile_each(acc, [&](int r, int c, double& v) { v = -t[c * kPP + r]; });
      dmma_tile<2, 2, kPP, kPP, 16>(acc, a + 16 * i, a + k * C);
      put(t, acc, -1.0);
    }
    __syncthreads();
  }
  if (warp < NB && 16 * warp < d)
    lu_inv16(fb + warp * B, d - 16 * warp, s_rcp + 16 * warp, li + warp * B, ui + warp * B);
  __syncthreads();
  // the off-diagonal block of an inverse of twice the size, from the halves'
  // inverses: -L22^{-1} (L21 L11^{-1}) and -(U11^{-1} U12) U22^{-1}; the product in
  // brackets goes through the block's own place
  if (warp < 4 && 32 * (warp & 1) + 16 < d) {  // 32: two blocks of L^{-1}, two of U^{-1}, one warp each
    const int o = 2 * (warp & 1) * B;
    double* x = warp < 2 ? li + o + 16 : ui + o + C;
    double acc[2][2][2] = {}, z[2][2][2] = {};
    if (warp < 2)
      dmma_tile<2, 2, kPP, kPP, 16>(acc, fb + o + 16, li + o);
    else
      dmma_tile<2, 2, kPP, kPP, 16>(acc, ui + o, fb + o + C);
    put(x, acc, 1.0);
    __syncwarp();
    if (warp < 2)
      dmma_tile<2, 2, kPP, kPP, 16>(z, li + o + B, x);
    else
      dmma_tile<2, 2, kPP, kPP, 16>(z, x, ui + o + B);
    __syncwarp();
    put(x, z, -1.0);
  }
  __syncthreads();
  if (d > 32) {  // 64: a 16 x 16 tile of the 32 x 32 block each, warps 0..3 of L^{-1}, 4..7 of U^{-1}
    const int i = 16 * (warp & 1), k = (warp & 2) * (C / 2);
    double* x = (warp < 4 ? li + 32 : ui + 2 * C) + i + k;
    double acc[2][2][2] = {}, z[2][2][2] = {};
    if (warp < 4)
      dmma_tile<2, 2, kPP, kPP, 32>(acc, fb + 32 + i, li + k);
    else
      dmma_tile<2, 2, kPP, kPP, 32>(acc, ui + i, fb + 2 * C + k);
    put(x, acc, 1.0);
    __syncthreads();
    if (warp < 4)
      dmma_tile<2, 2, kPP, kPP, 32>(z, li + 2 * B + i, li + 32 + k);
    else
      dmma_tile<2, 2, kPP, kPP, 32>(z, ui + 2 * C + i, ui + 2 * B + k);
    __syncthreads();
    put(x, z, -1.0);
  }
  __syncthreads();
  for (int e = tid; e < (d <= kDB ? kNP * kDB / 2 : kNP * kNP / 2); e += kNPT) {
    const int c = e >> 5, r = 2 * (e & 31), q = c * kPP + r;
    const double2 *f2 = reinterpret_cast<const double2*>(fb + q),
                  *l2 = reinterpret_cast<const double2*>(li + q),
                  *u2 = reinterpret_cast<const double2*>(ui + q);
    if (c < d && r < d) *reinterpret_cast<double2*>(D + (size_t)c * m + r) = *f2;
    if (S) {
      reinterpret_cast<double2*>(S)[e] = *l2;
      reinterpret_cast<double2*>(S + kNP * kNP)[e] = *u2;
    }
  }
  for (int b = 0; b * kDB < d; ++b) {
    const int nb = min(kDB, d - b * kDB), o = b * kDB;
    double* Lb = Di + (size_t)b * 2 * kDB * kDB;
    double* Ub = Lb + kDB * kDB;
    for (int e = tid; e < kDB * kDB; e += kNPT) {
      const int c = e / kDB, r = e - c * kDB;
      const double id = r == c ? 1.0 : 0.0;
      Lb[e] = (r < nb && c < nb) ? li[(o + c) * kPP + o + r] : id;
      Ub[e] = (r < nb && c < nb) ? ui[(o + c) * kPP + o + r] : id;
    }
  }
  return bad;
}

// Per leaf (leaves[blockIdx.x]) with m > K0: the diagonal block A[K0:K0+D,
// K0:K0+D], D = min(kOB2, m - K0), factored in place; scr and dinv receive the
// inverses of its 64 x 64 diagonal blocks (see lu_diag64).  Step j: the
// diagonal block, L_ij = A_ij U_jj^{-1} (multipliers checked), and per block
// column k U_jk = L_jj^{-1} A_jk and A_ik -= L_ij U_jk, all as 64 x 64 x 64
// products on the FP64 tensor cores from three staged blocks (104 KB, so two
// CTAs, or one and an update's, share an SM and fill each other's waits).
// One CTA for the whole block: the step's 64-column launches over all leaves
// that it replaces (diagonal, panel, update: 50 + 60 + 70 us each, four per
// outer block) streamed every leaf's 256 columns from HBM each time and left
// the SMs waiting between them.
constexpr size_t kNPBlockSmem = sizeof(double) * 3 * kNB2;

__global__ void __launch_bounds__(kNPT, 2) lu_np_block_kernel(
    const int* __restrict__ leaves, int K0, const int2* __restrict__ leaf_rng,
    const int64_t* __restrict__ blk_off, const int64_t* __restrict__ dinv_off, double* lu,
    double* __restrict__ dinv, double* __restrict__ scr, int* __restrict__ fail) {
  extern __shared__ __align__(16) double nsm[];
  __shared__ double s_rcp[kNP];  // reciprocal of each pivot
  chain_wait();  // the previous launch of the chain has finished
  chain_signal();
  double* b0 = nsm;              // L_jj^{-1}; then one of L_ij's two buffers
  double* b1 = nsm + kNB2;       // U_jj^{-1}; one of A_jk's two buffers; U_jk
  double* b2 = nsm + 2 * kNB2;   // A_ij; the other of A_jk's, of L_ij's buffers
  const int leaf = leaves[blockIdx.x];
  const int m = 2 * leaf_rng[leaf].y, D = min(kOB2, m - K0);
  double* A = lu + blk_off[leaf] + (size_t)K0 * m + K0;
  auto blk = [&](int i, int j) { return A + (size_t)(kNP * j) * m + kNP * i; };
  auto size = [&](int i) { return min(kNP, D - i * kNP); };
  const int tid = threadIdx.x, warp = tid >> 5;
  // this warp's 32 x 16 tile of a product; products with a triangular inverse
  // stop at its diagonal, and the tiles are dealt so that the four schedulers
  // (warp modulo 4) get equal parts of them
  const int r0 = 32 * ((warp ^ (warp >> 2)) & 1), c0 = 16 * (warp < 4 ? warp >> 1 : 5 - (warp >> 1));
  const int nb = (D + kNP - 1) / kNP;
  bool bad = false;
  for (int j = 0; j < nb; ++j) {
    bad |= lu_diag64(blk(j, j), m, size(j), b0, b1, b2, s_rcp,
                     m > K0 + kOB2 ? scr + ((size_t)blockIdx.x * (kOB2 / kNP) + j) * 2 * kNP * kNP
                                   : nullptr,
                     dinv + dinv_off[leaf] + (size_t)((K0 + j * kNP) / kDB) * 2 * kDB * kDB);
    // L_ij = A_ij U_jj^{-1}
    for (int i = j + 1; i < nb; ++i) {
      __syncthreads();
      stage64<kNPT>(b2, blk(i, j), m, size(i), kNP);
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
      double acc[4][2][2] = {};
      dmma_tile_part<4, 2, kPP, kPP>(acc, b2 + r0, b1 + c0 * kPP, c0 + 16);
      double* out = blk(i, j);
      tile_each(acc, [&](int r, int c, double v) {
        if (r0 + r < size(i)) {
          if (!(fabs(v) <= kNoPivBound)) bad = true;
          out[(size_t)(c0 + c) * m + r0 + r] = v;
        }
      });
    }
    // U_jk = L_jj^{-1} A_jk, A_jk one block ahead in b1 and b2
    __syncthreads();
    if (j + 1 < nb) {
      stage64<kNPT>(b1, blk(j, j + 1), m, kNP, size(j + 1));
      cp_async_commit();
    }
    for (int k = j + 1; k < nb; ++k) {
      cp_async_wait<0>();
      __syncthreads();
      if (k + 1 < nb) {
        stage64<kNPT>((k - j) & 1 ? b2 : b1, blk(j, k + 1), m, kNP, size(k + 1));
        cp_async_commit();
      }
      double acc[4][2][2] = {};
      dmma_tile_part<4, 2, kPP, kPP>(acc, b0 + r0, ((k - j) & 1 ? b1 : b2) + c0 * kPP, r0 + 32);
      double* out = blk(j, k);
      tile_each(acc, [&](int r, int c, double v) {
        if (c0 + c < size(k)) out[(size_t)(c0 + c) * m + r0 + r] = v;
      });
    }
    // A_ik -= L_ij U_jk, L_ij one block ahead in b0 and b2
    __syncthreads();
    int buf = 0;
    for (int k = j + 1; k < nb; ++k) {
      if (k > j + 1) __syncthreads();  // b1 is read
      stage64<kNPT>(b1, blk(j, k), m, kNP, size(k));
      if (k == j + 1) stage64<kNPT>(b0, blk(j + 1, j), m, size(j + 1), kNP);
      cp_async_commit();
      for (int i = j + 1; i < nb; ++i, buf ^= 1) {
        double acc[4][2][2];
        double* out = blk(i, k);
        tile_each(acc, [&](int r, int c, double& v) {
          v = r0 + r < size(i) && c0 + c < size(k) ? -out[(size_t)(c0 + c) * m + r0 + r] : 0.0;
        });
        cp_async_wait<0>();
        __syncthreads();
        const int in = i + 1 < nb ? i + 1 : j + 1;  // the next block of the cycle over i
        if (i + 1 < nb || k + 1 < nb) {
          stage64<kNPT>(buf ? b0 : b2, blk(in, j), m, size(in), kNP);
          cp_async_commit();
        }
        dmma_tile<4, 2, kPP, kPP, kNP>(acc, (buf ? b2 : b0) + r0, b1 + c0 * kPP);
        tile_each(acc, [&](int r, int c, double v) {
          if (r0 + r < size(i) && c0 + c < size(k)) out[(size_t)(c0 + c) * m + r0 + r] = -v;
        });
      }
    }
    __syncthreads();
  }
  if (__syncthreads_or(bad) && tid == 0) fail[leaf] = 1;
}

// item = (leaf, slot, kind, off) of a leaf with m > K0 + kOB2: kind 0, rows
// [off, off + 64) of L21; kind 1, columns [off, off + 64) of U12.  slot = the
// leaf's position in the block kernel's launch (its scratch).  The chunk lies
// in shared memory, the 64 x 64 blocks of the diagonal block's factors and
// inverses pass through one buffer (104 KB together, so that two CTAs share
// an SM and fill each other's waits):
//   kind 0: Y_j = Y_j U_jj^{-1}, then Y_i -= Y_j U_ji for i > j (columns by 64),
//   kind 1: X_j = L_jj^{-1} X_j, then X_i -= L_ij X_j for i > j (rows by 64).
constexpr int kTP1 = kOB2 + 4;  // kind 1: pitch of a column of the chunk
constexpr size_t kNPBorderSmem = sizeof(double) * (kOB2 * kPP + kNB2);

template <int KIND>
__device__ __forceinline__ bool lu_border(double* T, double* f, double* A, int m, int K0,
                                          int off, const double* S) {
  constexpr int NB = kOB2 / kNP;
  const int cnt = min(kNP, m - off);
  double* chunk = KIND == 0 ? A + (size_t)K0 * m + off : A + (size_t)off * m + K0;
  const double* F = A + (size_t)K0 * m + K0;  // the factored diagonal block
  // this warp's 32 x 16 tile of a 64 x 64 product (dealt as in the block kernel)
  const int warp = threadIdx.x >> 5;
  const int r0 = 32 * ((warp ^ (warp >> 2)) & 1), c0 = 16 * (warp < 4 ? warp >> 1 : 5 - (warp >> 1));
  auto stage_factor = [&](int i, int j) {
    if (i == j)
      stage64<kNPT>(f, S + (size_t)j * 2 * kNP * kNP + (KIND == 0 ? kNP * kNP : 0), kNP, kNP,
                    kNP);
    else if (KIND == 0)
      stage64<kNPT>(f, F + (size_t)(kNP * i) * m + kNP * j, m, kNP, kNP);
    else
      stage64<kNPT>(f, F + (size_t)(kNP * j) * m + kNP * i, m, kNP, kNP);
    cp_async_commit();
  };
  if (KIND == 0) {
#pragma unroll
    for (int j = 0; j < NB; ++j)
      stage64<kNPT>(T + j * kNB2, chunk + (size_t)(j * kNP) * m, m, cnt, kNP);
  } else {
#pragma unroll
    for (int e = 0; e < kNP * kOB2 / 2 / kNPT; ++e) {
      const int q = (int)threadIdx.x + kNPT * e, c = q / (kOB2 / 2), r = 2 * (q % (kOB2 / 2));
      const bool ok = c < cnt;
      cp_async16(T + c * kTP1 + r, ok ? chunk + (size_t)c * m + r : chunk, ok);
    }
  }
  // entry (r, c) of the warp's tile in block i of the chunk
  auto at = [&](int i, int r, int c) -> double& {
    return KIND == 0 ? T[i * kNB2 + (c0 + c) * kPP + r0 + r]
                     : T[(c0 + c) * kTP1 + i * kNP + r0 + r];
  };
  auto multiply = [&](double (&acc)[4][2][2], int j, bool tri) {
    if ((KIND == 0 ? r0 : c0) >= cnt) return;  // past the chunk's edge
    if (KIND == 0) {
      if (tri)
        dmma_tile_part<4, 2, kPP, kPP>(acc, T + j * kNB2 + r0, f + c0 * kPP, c0 + 16);
      else
        dmma_tile<4, 2, kPP, kPP, kNP>(acc, T + j * kNB2 + r0, f + c0 * kPP);
    } else {
      if (tri)
        dmma_tile_part<4, 2, kPP, kTP1>(acc, f + r0, T + c0 * kTP1 + j * kNP, r0 + 32);
      else
        dmma_tile<4, 2, kPP, kTP1, kNP>(acc, f + r0, T + c0 * kTP1 + j * kNP);
    }
  };
  bool bad = false;
  for (int j = 0; j < NB; ++j)
    for (int i = j; i < NB; ++i) {
      if (i + j > 0) __syncthreads();  // the buffer is read, the chunk written
      stage_factor(i, j);
      cp_async_wait<0>();
      __syncthreads();
      double acc[4][2][2] = {};
      if (i == j) {
        multiply(acc, j, true);
        __syncthreads();  // block j is read
        tile_each(acc, [&](int r, int c, double v) {
          if (KIND == 0 && !(fabs(v) <= kNoPivBound)) bad = true;
          at(j, r, c) = v;
        });
      } else {
        tile_each(acc, [&](int r, int c, double& v) { v = -at(i, r, c); });
        multiply(acc, j, false);
        tile_each(acc, [&](int r, int c, double v) { at(i, r, c) = -v; });
      }
    }
  __syncthreads();
  for (int q = threadIdx.x; q < kNP * kOB2; q += kNPT) {
    const int c = KIND == 0 ? q / kNP : q / kOB2, r = KIND == 0 ? q % kNP : q % kOB2;
    if (KIND == 0 ? r < cnt : c < cnt)
      chunk[(size_t)c * m + r] = T[c * (KIND == 0 ? kPP : kTP1) + r];
  }
  return bad;
}

__global__ void __launch_bounds__(kNPT, 2) lu_np_border_kernel(
    const int4* __restrict__ items, int K0, const int2* __restrict__ leaf_rng,
    const int64_t* __restrict__ blk_off, double* lu, const double* __restrict__ scr,
    int* __restrict__ fail) {
  extern __shared__ __align__(16) double nsm[];
  chain_wait();  // the previous launch of the chain has finished
  chain_signal();
  const int4 it = items[blockIdx.x];
  const int m = 2 * leaf_rng[it.x].y;
  double* A = lu + blk_off[it.x];
  const double* S = scr + (size_t)it.y * (kOB2 / kNP) * 2 * kNP * kNP;
  double* f = nsm + kOB2 * kPP;
  const bool bad = it.z == 0 ? lu_border<0>(nsm, f, A, m, K0, it.w, S)
                             : lu_border<1>(nsm, f, A, m, K0, it.w, S);
  if (__syncthreads_or(bad) && threadIdx.x == 0) fail[it.x] = 1;
}

// Updates of the unpivoted factorisation: item = (leaf, r0, c0, -):
// C = A[r0:r0+128, c0:c0+64] -= A[r0:, k0:k0+kd] A[k0:k0+kd, c0:] with
// kd = min(kdepth, m - k0), rows and columns clipped at m.  FP64 tensor cores, a
// 32 x 32 tile per warp: -C is loaded into the accumulators, the products are added
// in order of k, and the negative of the sum is stored.  16-deep slices of L
// (k-major) and U (by column) arrive by cp.async in a ring of four (zero-filled
// outside the tile: m, r0, c0, k0 and the depth are even, so a 16-byte chunk is
// wholly inside or outside), with one barrier per slice: three slices are in
// flight while one is multiplied.  Two 32-deep slices and two barriers each took
// 579 us instead of 562 at depth 128 and 400 instead of 372 at depth 64 (31 leaves
// of order ~1400).  The form with 8 x 4 outputs per thread on DFMA
// was bound by its 12 shared-load words per 32 multiply-adds: 45-50 % of the
// FP64 pipe.
constexpr int kG2M = 128, kG2N = 64, kG2K = 16;
constexpr int kG2LP = kG2M + 4;  // L slice: pitch of a depth's 128 rows
constexpr int kG2UP = kG2K + 4;  // U slice: pitch of a column's depths
constexpr int kG2S = 4;           // slices in the ring
constexpr size_t kGemm2Smem = sizeof(double) * kG2S * (kG2K * kG2LP + kG2N * kG2UP);

__global__ void __launch_bounds__(256, 2) lu_gemm2_kernel(const int4* __restrict__ items, int k0,
                                                          int kdepth,
                                                          const int2* __restrict__ leaf_rng,
                                                          const int64_t* __restrict__ blk_off,
                                                          double* __restrict__ lu) {
  extern __shared__ __align__(16) double gsm2[];
  chain_wait();  // the previous launch of the chain has finished
  chain_signal();
  double* sL = gsm2;                      // [kG2S][kG2K][kG2LP]  L slices, k-major
  double* sU = gsm2 + kG2S * kG2K * kG2LP;  // [kG2S][kG2N][kG2UP]  U slices, by column
  const int4 it = items[blockIdx.x];
  const int leaf = it.x, r0 = it.y, c0 = it.z;
  const int m = 2 * leaf_rng[leaf].y;
  const int kd = min(kdepth, m - k0);
  double* A = lu + blk_off[leaf];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto load_slice = [&](int kc, int buf) {
    const int nbk = min(kG2K, kd - kc), kb = k0 + kc;
    double* L = sL + buf * kG2K * kG2LP;
    double* U = sU + buf * kG2N * kG2UP;
#pragma unroll
    for (int e = 0; e < (kG2K * kG2M / 2) / 256; ++e) {
      const int q = tid + 256 * e;
      const int k = q / (kG2M / 2), rr = 2 * (q % (kG2M / 2));
      const bool ok = k < nbk && r0 + rr < m;
      cp_async16(L + k * kG2LP + rr, ok ? A + (size_t)(kb + k) * m + r0 + rr : A, ok);
    }
    // U by column (the source's own layout): 16-byte chunks of 2 k
#pragma unroll
    for (int e = 0; e < (kG2K * kG2N / 2) / 256; ++e) {
      const int q = tid + 256 * e;
      const int c = q / (kG2K / 2), kk = 2 * (q % (kG2K / 2));
      const bool ok = kk < nbk && c0 + c < m;
      cp_async16(U + c * kG2UP + kk, ok ? A + (size_t)(c0 + c) * m + kb + kk : A, ok);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
#pragma unroll
  for (int p = 0; p < kG2S - 1; ++p) {
    if (p * kG2K < kd) load_slice(p * kG2K, p);
    else asm volatile("cp.async.commit_group;\n" ::);
  }
  // this warp's tile, and the lane's row and column in it
  const int wr = 32 * (warp & 3), wc = 32 * (warp >> 2);
  const int rl = r0 + wr + (lane >> 2), cl = c0 + wc + 2 * (lane & 3);
  double acc[4][4][2];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int c = cl + 8 * q + b;
      const double* cc = A + (size_t)min(c, m - 1) * m;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = rl + 8 * i;
        acc[i][q][b] = (c < m && r < m) ? -cc[r] : 0.0;
      }
    }
  for (int kc = 0, buf = 0; kc < kd; kc += kG2K, buf = (buf + 1) & (kG2S - 1)) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kG2S - 2));
    __syncthreads();
    if (kc + (kG2S - 1) * kG2K < kd) load_slice(kc + (kG2S - 1) * kG2K, (buf + kG2S - 1) & (kG2S - 1));
    else asm volatile("cp.async.commit_group;\n" ::);
    if (r0 + wr < m && c0 + wc < m)
      dmma_tile<4, 4, kG2LP, kG2UP, kG2K>(acc, sL + buf * kG2K * kG2LP + wr,
                                          sU + buf * kG2N * kG2UP + wc * kG2UP);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int c = cl + 8 * q + b;
      if (c >= m) continue;
      double* cc = A + (size_t)c * m;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = rl + 8 * i;
        if (r < m) cc[r] = -acc[i][q][b];
      }
    }
}

// every leaf: no interchange (1-based local pivots i + 1) and the identity
// row permutation of the applies
__global__ void lu_np_identity_kernel(const int2* __restrict__ leaf_rng, int* __restrict__ piv,
                                      int* __restrict__ perm) {
  const int2 lr = leaf_rng[blockIdx.x];
  const int m = 2 * lr.y;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    piv[2 * lr.x + i] = i + 1;
    perm[2 * lr.x + i] = i;
  }
}

__global__ void diag_kernel(const double* r, double* z, int n, double s1, double s2) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) z[i] = r[i] / s1;
  else if (i < 2 * n) z[i] = r[i] / s2;
}

// the leaf blocks' kernel values for the given (leaf, column) tiles
void launch_assemble(Handle& H, const int2* tiles, int ntiles, cudaStream_t s) {
  Tree& T = H.tree;
  double rad = 0.0;
  for (int c : T.leaves) rad = std::max(rad, T.rad[c]);
  TABI_K(K_ASSEMBLE, s);
  // no two faces of a leaf are further apart than its diameter
  (H.prm.kappa * 2.0 * rad < 0.99 * kExpTabEnd ? assemble_kernel<false> : assemble_kernel<true>)<<<
      ntiles, 256, 0, s>>>(tiles, T.d_leaf_rng.p, T.d_blk_off.p, H.d_x.p, H.d_y.p, H.d_z.p,
                           H.d_nx.p, H.d_ny.p, H.d_nz.p, H.d_area.p, H.prm.kappa,
                           H.prm.eps1 / H.prm.eps0, T.d_lu.p);
}

}  // namespace

void build_precond(Handle& H, cudaStream_t s) {
  Tree& T = H.tree;
  if (H.prm.iprcd != 1) {
    H.has_precond = true;
    return;
  }
  const int nl = T.nleaf;
  std::vector<int2> rng(nl);
  T.blk_off.resize(nl);
  int64_t off = 0;
  PinVec<int2>& tiles = H.pc_h_tiles;
  tiles.restart();
  for (int l = 0; l < nl; ++l) {
    int c = T.leaves[l];
    rng[l] = make_int2(T.ibeg[c], T.num[c]);
    T.blk_off[l] = off;
    off += 4LL * T.num[c] * T.num[c];
    for (int j = 0; j < T.num[c]; j += kAsmCols) tiles.push(make_int2(l, j));
  }
  T.d_lu.alloc(std::max<int64_t>(off, 1));
  T.d_piv.alloc(2 * (size_t)H.n);
  T.d_blk_off.alloc(nl);
  T.d_leaf_rng.alloc(nl);
  DBuf<int2>& d_tiles = H.pc_tiles;
  d_tiles.alloc(tiles.len);
  DBuf<int>& d_info = H.pc_info;
  d_info.alloc(nl);
  H.pc_h_blk_off.assign(T.blk_off.data(), nl);
  H.pc_h_blk_off.upload(T.d_blk_off, s);
  H.pc_h_rng.assign(rng.data(), nl);
  H.pc_h_rng.upload(T.d_leaf_rng, s);
  tiles.upload(d_tiles, s);
  double eps = H.prm.eps1 / H.prm.eps0;
  launch_assemble(H, d_tiles.p, (int)tiles.len, s);
  TABI_CUDA(cudaMemsetAsync(d_info.p, 0, sizeof(int) * nl, s));
  // apply lists (they depend on the leaf sizes only, so they are built while
  // the assembly runs): blocks of order > kSolveSmall and the others, on the side
  // stream (see solve_kernel); largest first in each
  {
    std::vector<int> big, small;
    for (int l = 0; l < nl; ++l) (2 * rng[l].y > kSolveSmall ? big : small).push_back(l);
    const int64_t bytes = (int64_t)sizeof(double) * off;  // of all factors
    T.solve_rows = nl > 1 ? bytes <= kRowBytes
                          : bytes <= kLoneBytes || (rng[0].y % 2 && 2 * rng[0].y <= kLoneOrder);
    std::sort(big.begin(), big.end(), [&](int a, int b) { return rng[a].y > rng[b].y; });
    std::sort(small.begin(), small.end(), [&](int a, int b) { return rng[a].y > rng[b].y; });
    T.n_solve_big = (int)big.size();
    T.n_solve_small = (int)small.size();
    big.insert(big.end(), small.begin(), small.end());
    H.pc_h_solve_list.assign(big.data(), big.size());
    H.pc_h_solve_list.upload(T.d_solve_list, s);
  }
  // ---- unpivoted factorisation of every leaf, certified (see lu_np_block_kernel)
  H.pc_lu_phase.emplace(H.prof, K_PHASE_LU, s);
  const bool try_np = (H.prm.flags & TABI_FLAG_PIVOTED_LU) == 0;
  if (try_np) {
    DBuf<int>& d_fail = H.pc_fail;
    d_fail.alloc(nl);
    TABI_CUDA(cudaMemsetAsync(d_fail.p, 0, sizeof(int) * nl, s));
    T.d_lu_perm.alloc(2 * (size_t)H.n);
    { TABI_K(K_LU_POST, s); lu_np_identity_kernel<<<nl, 256, 0, s>>>(T.d_leaf_rng.p, T.d_piv.p, T.d_lu_perm.p); }
    // the inverse diagonal blocks are written by the diagonal kernel
    T.dinv_off.resize(nl);
    int64_t doff = 0;
    for (int l = 0; l < nl; ++l) {
      T.dinv_off[l] = doff;
      doff += (int64_t)ceil_div(2 * rng[l].y, kDB) * 2 * kDB * kDB;
    }
    T.d_dinv.alloc(std::max<int64_t>(doff, 1));
    T.d_dinv_off.alloc(nl);
    H.pc_h_dinv_off.assign(T.dinv_off.data(), nl);
    H.pc_h_dinv_off.upload(T.d_dinv_off, s);
    raise_smem_limit((const void*)lu_np_block_kernel, kNPBlockSmem);
    raise_smem_limit((const void*)lu_np_border_kernel, kNPBorderSmem);
    raise_smem_limit((const void*)lu_gemm2_kernel, kGemm2Smem);
    std::vector<int> grp[2];
    for (int l = 0; l < nl; ++l) grp[2 * rng[l].y > kLuSmallBlock ? 0 : 1].push_back(l);
    for (auto& g : grp)
      std::sort(g.begin(), g.end(), [&](int a, int b) { return rng[a].y > rng[b].y; });
    // both groups on the handle's high-priority LU streams, forked from s
    TABI_CUDA(cudaEventRecord(H.ev_fork, s));
    TABI_CUDA(cudaStreamWaitEvent(H.lu_hi, H.ev_fork, 0));
    TABI_CUDA(cudaStreamWaitEvent(H.lu_small, H.ev_fork, 0));
    // Right-looking order in outer blocks of kOB2 columns: the diagonal block of
    // every leaf, its L21 and U12 chunks, the trailing update.
    //
    // Look-ahead (the large-block group): the trailing update of an outer block
    // is split.  The next outer block's rows and columns are updated on the
    // group's stream, the rest on the middle-priority auxiliary stream, beside
    // the next block's factorisation and chunks, which need only the former.
    // The next block's own update waits for the auxiliary stream.
    struct Launch {
      // 0 diagonal block, 1 its chunks, 2 update, 3 fork to the auxiliary
      // stream, 4 wait for the auxiliary stream, 5 update on the auxiliary stream
      int kind;
      int k0, off, cnt;
    };
    // one group's plan: item lists (uploaded on st) and its launches
    auto plan_np = [&](const std::vector<int>& order, Handle::NpPlan& B, cudaStream_t st,
                       bool la) {
      int gmax = 0;
      for (int l : order) gmax = std::max(gmax, 2 * rng[l].y);
      std::vector<Launch> plan;
      PinVec<int>& dl = B.h_dleaves;
      PinVec<int4>& pit = B.h_pitems;
      PinVec<int4>& git = B.h_gitems;
      dl.restart();
      pit.restart();
      git.restart();
      auto emit = [&](int kind, int k0, size_t before, size_t after) {
        if (after > before) plan.push_back({kind, k0, (int)before, (int)(after - before)});
      };
      bool rest_pending = false;  // an update on the auxiliary stream not yet waited for
      for (int K0 = 0; K0 < gmax; K0 += kOB2) {
        const int Kend = K0 + kOB2, Knext = la ? Kend + kOB2 : INT_MAX;
        const size_t d0 = dl.len, p0 = pit.len, g0 = git.len;
        int slot = 0;
        for (int l : order) {
          const int m = 2 * rng[l].y;
          if (m <= K0) continue;
          dl.push(l);
          for (int off = Kend; off < m; off += kNP) {
            pit.push(make_int4(l, slot, 0, off));
            pit.push(make_int4(l, slot, 1, off));
          }
          for (int r0 = Kend; r0 < m; r0 += kG2M)
            for (int c0 = Kend; c0 < m && (r0 < Knext || c0 < Knext); c0 += kG2N)
              git.push(make_int4(l, r0, c0, 0));
          ++slot;
        }
        const size_t g1 = git.len;
        for (int l : order) {
          const int m = 2 * rng[l].y;
          for (int r0 = Knext; la && r0 < m; r0 += kG2M)
            for (int c0 = Knext; c0 < m; c0 += kG2N) git.push(make_int4(l, r0, c0, 0));
        }
        emit(0, K0, d0, dl.len);
        emit(1, K0, p0, pit.len);
        if (git.len > g1) plan.push_back({3, K0, 0, 0});
        if (rest_pending) plan.push_back({4, K0, 0, 0});
        emit(2, K0, g0, g1);
        rest_pending = git.len > g1;
        emit(5, K0, g1, git.len);
      }
      if (rest_pending) plan.push_back({4, gmax, 0, 0});
      dl.upload(B.dleaves, st);
      pit.upload(B.pitems, st);
      git.upload(B.gitems, st);
      B.scr.alloc(order.size() * (kOB2 / kNP) * 2 * kNP * kNP);
      return plan;
    };
    // Issues launch `at` of a group's plan.  Kernels follow kernels on the
    // group's stream as a programmatic chain; the first one after the uploads
    // or a cross-stream event starts the ordinary way.
    struct Issuer {
      std::vector<Launch> plan;
      Handle::NpPlan* B;
      cudaStream_t st;
      size_t at = 0;
      bool chain = false;
    };
    auto issue_one = [&](Issuer& is) {
      const Launch& q = is.plan[is.at++];
      Handle::NpPlan& B = *is.B;
      cudaStream_t st = is.st;
      bool& chain = is.chain;
      {
        if (q.kind == 0) {
          TABI_K(K_LU, st);
          launch_chained(chain, lu_np_block_kernel, dim3(q.cnt), dim3(kNPT), kNPBlockSmem, st,
                         B.dleaves.p + q.off, q.k0, T.d_leaf_rng.p, T.d_blk_off.p,
                         T.d_dinv_off.p, T.d_lu.p, T.d_dinv.p, B.scr.p, d_fail.p);
          chain = true;
        } else if (q.kind == 1) {
          TABI_K(K_LU_STRIP, st);
          launch_chained(chain, lu_np_border_kernel, dim3(q.cnt), dim3(kNPT), kNPBorderSmem, st,
                         B.pitems.p + q.off, q.k0, T.d_leaf_rng.p, T.d_blk_off.p, T.d_lu.p,
                         B.scr.p, d_fail.p);
          chain = true;
        } else if (q.kind == 3) {
          TABI_CUDA(cudaEventRecord(H.ev_la, st));
          TABI_CUDA(cudaStreamWaitEvent(H.aux, H.ev_la, 0));
          chain = false;
        } else if (q.kind == 4) {
          TABI_CUDA(cudaStreamWaitEvent(st, H.ev_rest, 0));
          chain = false;
        } else {
          cudaStream_t gs = q.kind == 5 ? H.aux : st;
          TABI_K(K_LU_UPDATE, gs);
          launch_chained(chain && q.kind == 2, lu_gemm2_kernel, dim3(q.cnt), dim3(256),
                         kGemm2Smem, gs,
                         B.gitems.p + q.off, q.k0, kOB2, T.d_leaf_rng.p, T.d_blk_off.p,
                         T.d_lu.p);
          if (q.kind == 5) TABI_CUDA(cudaEventRecord(H.ev_rest, H.aux));
          else chain = true;
        }
      }
    };
    // both plans first, then their launches interleaved, so that both chains
    // start at once (the host issues far faster than the GPU runs them)
    Issuer big{}, small{};
    big.B = &H.pc_np[0];
    big.st = H.lu_hi;
    small.B = &H.pc_np[1];
    small.st = H.lu_small;
    if (!grp[0].empty()) big.plan = plan_np(grp[0], H.pc_np[0], H.lu_hi, true);
    if (!grp[1].empty()) small.plan = plan_np(grp[1], H.pc_np[1], H.lu_small, false);
    while (big.at < big.plan.size() || small.at < small.plan.size()) {
      if (big.at < big.plan.size()) issue_one(big);
      if (small.at < small.plan.size()) issue_one(small);
    }
  }
}

void finish_precond(Handle& H, cudaStream_t s) {
  if (H.prm.iprcd != 1 || H.has_precond) return;
  Tree& T = H.tree;
  const int nl = T.nleaf;
  std::vector<int2> rng(nl);
  for (int l = 0; l < nl; ++l) {
    const int c = T.leaves[l];
    rng[l] = make_int2(T.ibeg[c], T.num[c]);
  }
  const double eps = H.prm.eps1 / H.prm.eps0;
  DBuf<int>& d_info = H.pc_info;
  const bool try_np = (H.prm.flags & TABI_FLAG_PIVOTED_LU) == 0;
  // Two leaf groups with plans of their own: blocks of order above
  // kLuSmallBlock and the others, so the many short factorisations of small
  // leaves run beside the long chain of steps of the large ones instead of
  // inside its launches.  The unpivoted factorisation runs them on the
  // handle's LU streams (see below); the pivoted one on the caller's stream
  // and the side stream, with one fork after the assembly and one join at
  // the end (fork / join).
  auto fork = [&](bool split) {
    if (!split) return;
    TABI_CUDA(cudaEventRecord(H.ev_fork, s));
    TABI_CUDA(cudaStreamWaitEvent(H.side, H.ev_fork, 0));
  };
  auto join = [&](bool split) {
    if (!split) return;
    TABI_CUDA(cudaEventRecord(H.ev_join, H.side));
    TABI_CUDA(cudaStreamWaitEvent(s, H.ev_join, 0));
  };
  std::vector<int> pv_leaves;  // leaves factored with partial pivoting
  if (try_np) {
    DBuf<int>& d_fail = H.pc_fail;
    TABI_CUDA(cudaEventRecord(H.ev_join, H.lu_small));
    TABI_CUDA(cudaStreamWaitEvent(s, H.ev_join, 0));
    TABI_CUDA(cudaEventRecord(H.ev_lu_join, H.lu_hi));
    TABI_CUDA(cudaStreamWaitEvent(s, H.ev_lu_join, 0));
    std::vector<int> failed(nl);
    TABI_CUDA(cudaMemcpyAsync(failed.data(), d_fail.p, sizeof(int) * nl, cudaMemcpyDeviceToHost,
                              s));
    TABI_CUDA(cudaStreamSynchronize(s));
    for (int l = 0; l < nl; ++l)
      if (failed[l]) pv_leaves.push_back(l);
    if (!pv_leaves.empty()) {
      // those blocks again from their kernel values
      std::vector<int2> ptiles;
      for (int l : pv_leaves)
        for (int j = 0; j < rng[l].y; j += kAsmCols) ptiles.push_back(make_int2(l, j));
      H.pc_tiles2.alloc(ptiles.size());
      TABI_CUDA(cudaMemcpyAsync(H.pc_tiles2.p, ptiles.data(), sizeof(int2) * ptiles.size(),
                                cudaMemcpyHostToDevice, s));
      launch_assemble(H, H.pc_tiles2.p, (int)ptiles.size(), s);
    }
  } else {
    for (int l = 0; l < nl; ++l) pv_leaves.push_back(l);
  }
  H.pc_pv_leaves = (int)pv_leaves.size();
  if (!pv_leaves.empty()) {
    // batched LU for blocks with m <= kPanelMaxM; the global-memory kernel for
    // larger ones
    int mmax = 0;
    bool any_big = false;
    std::vector<int> big_leaves;
    for (int l : pv_leaves) {
      int m = 2 * rng[l].y;
      if (m <= kPanelMaxM) mmax = std::max(mmax, m);
      else {
        any_big = true;
        big_leaves.push_back(l);
      }
    }
    if (mmax > 0) {
      size_t smem = sizeof(double) * (size_t)mmax * kSP;
      raise_smem_limit((const void*)lu_panel_kernel, std::max<size_t>(smem, 48 * 1024));
    }
    raise_smem_limit((const void*)lu_gemm_kernel, kGemmSmem);
    // Two leaf groups with plans of their own: blocks of order above
    // kLuSmallBlock on the handle's stream, the others on its side stream, so
    // the many short factorisations of small leaves run beside the long
    // panel chain of the large ones instead of inside its launches; one fork
    // after the assembly, one join at the end.
    std::vector<int> grp[2];
    for (int l : pv_leaves) {
      const int m = 2 * rng[l].y;
      if (m <= kPanelMaxM) grp[m > kLuSmallBlock ? 0 : 1].push_back(l);
    }
    for (auto& g : grp)
      std::sort(g.begin(), g.end(), [&](int a, int b) { return rng[a].y > rng[b].y; });
    const bool split = H.side != nullptr && !grp[0].empty() && !grp[1].empty();
    fork(split);
    // Two-level right-looking LU (LAPACK DGETRF order) of one group.  Outer
    // blocks of kOB columns; inside one, 32-column panel steps update only
    // the block's own columns (and swap the columns left of the panel).  After
    // the block its kOB row interchanges are applied at once to the columns
    // right of it, U12 follows by 32-row TRSM + small GEMM steps, and the
    // trailing matrix gets one kOB-deep update.
    auto run_group = [&](const std::vector<int>& order, Handle::LuPlan& B, cudaStream_t st) {
      int gmax = 0;
      for (int l : order) gmax = std::max(gmax, 2 * rng[l].y);
      struct Launch {
        int kind;  // 0 panel, 1 strip, 2 gemm, 3 swap map, 4 row swap
        int k0, kdepth, off, cnt;
      };
      std::vector<Launch> plan;
      std::vector<int> pitems, mleaves;
      std::vector<int4> sitems, gitems, ritems;
      auto emit = [&](int kind, int k0, int kdepth, size_t before, size_t after) {
        if (after > before) plan.push_back({kind, k0, kdepth, (int)before, (int)(after - before)});
      };
      const auto pack = [](int re, int ce) { return (re << 16) | ce; };
      for (int K0 = 0; K0 < gmax; K0 += kOB) {
        for (int k0 = K0; k0 < std::min(gmax, K0 + kOB); k0 += kBP) {
          size_t p0 = pitems.size(), s0 = sitems.size(), g0 = gitems.size();
          for (int l : order) {
            const int m = 2 * rng[l].y;
            if (m <= k0) continue;
            pitems.push_back(l);
            const int nb = std::min(kBP, m - k0), ce = std::min(m, K0 + kOB);
            // left of the panel inside the outer block (the columns left of
            // the block get the block's swaps at its end)
            for (int c0 = K0; c0 < k0; c0 += kUC)
              sitems.push_back(make_int4(l, c0, std::min(c0 + kUC, k0), 0));
            for (int c0 = k0 + nb; c0 < ce; c0 += kUC)
              sitems.push_back(make_int4(l, c0, std::min(c0 + kUC, ce), 1));
            for (int r0 = k0 + nb; r0 < m; r0 += kGT)
              for (int c0 = k0 + nb; c0 < ce; c0 += kGT)
                gitems.push_back(make_int4(l, r0, c0, pack(m, ce)));
          }
          emit(0, k0, 0, p0, pitems.size());
          emit(1, k0, 0, s0, sitems.size());
          emit(2, k0, kBP, g0, gitems.size());
        }
        // the block's row interchanges on the columns left of it and right of it
        const int Kend = K0 + kOB;
        size_t m0 = mleaves.size(), r0i = ritems.size();
        for (int l : order) {
          const int m = 2 * rng[l].y;
          if (m <= K0 || (K0 == 0 && m <= Kend)) continue;
          const int slot = (int)(mleaves.size() - m0);
          mleaves.push_back(l);
          for (int c0 = 0; c0 < K0; c0 += kUC)
            ritems.push_back(make_int4(slot, c0, std::min(c0 + kUC, K0), l));
          for (int c0 = Kend; c0 < m; c0 += kUC)
            ritems.push_back(make_int4(slot, c0, std::min(c0 + kUC, m), l));
        }
        emit(3, K0, 0, m0, mleaves.size());
        emit(4, K0, 0, r0i, ritems.size());
        for (int kb = K0; kb < Kend; kb += kBP) {
          size_t s0 = sitems.size(), g0 = gitems.size();
          for (int l : order) {
            const int m = 2 * rng[l].y;
            if (m <= Kend) continue;
            for (int c0 = Kend; c0 < m; c0 += kUC)
              sitems.push_back(make_int4(l, c0, std::min(c0 + kUC, m), 3));
            for (int rr = kb + kBP; rr < Kend; rr += kGT)
              for (int c0 = Kend; c0 < m; c0 += kGT)
                gitems.push_back(make_int4(l, rr, c0, pack(Kend, m)));
          }
          emit(1, kb, 0, s0, sitems.size());
          emit(2, kb, kBP, g0, gitems.size());
        }
        size_t g0 = gitems.size();
        for (int l : order) {
          const int m = 2 * rng[l].y;
          if (m <= Kend) continue;
          for (int rr = Kend; rr < m; rr += kGT)
            for (int c0 = Kend; c0 < m; c0 += kGT) gitems.push_back(make_int4(l, rr, c0, 0));
        }
        emit(2, K0, kOB, g0, gitems.size());
      }
      auto up = [&](auto& buf, const auto& v) {
        buf.alloc(std::max<size_t>(v.size(), 1));
        if (!v.empty())
          TABI_CUDA(cudaMemcpyAsync(buf.p, v.data(), sizeof(v[0]) * v.size(),
                                    cudaMemcpyHostToDevice, st));
      };
      up(B.list, pitems);
      up(B.items, sitems);
      up(B.gitems, gitems);
      up(B.mleaves, mleaves);
      up(B.ritems, ritems);
      size_t maxm = 1;
      for (const Launch& L : plan)
        if (L.kind == 3) maxm = std::max<size_t>(maxm, (size_t)L.cnt);
      B.map.alloc(maxm * (4 * kOB + 1));
      for (const Launch& L : plan) {
        switch (L.kind) {
          case 0: {
            // the register-resident panel up to 512 x kRegMaxRows rows left
            // (the fewest warps that hold the rows, one row per thread below
            // 257 rows), the shared-memory one above; a launch is sized by its
            // first (largest) block
            const int mr = 2 * rng[pitems[L.off]].y - L.k0;
            const int* list = B.list.p + L.off;
            TABI_K(K_LU, st);
            if (mr <= 256)
              lu_panel_reg_kernel<256, 1><<<L.cnt, 256, 0, st>>>(
                  list, L.k0, T.d_leaf_rng.p, T.d_blk_off.p, T.d_lu.p, T.d_piv.p, d_info.p);
            else if (mr <= 512)
              lu_panel_reg_kernel<256, 2><<<L.cnt, 256, 0, st>>>(
                  list, L.k0, T.d_leaf_rng.p, T.d_blk_off.p, T.d_lu.p, T.d_piv.p, d_info.p);
            else if (mr <= 512 * kRegMaxRows)
              lu_panel_reg_kernel<512, kRegMaxRows><<<L.cnt, 512, 0, st>>>(
                  list, L.k0, T.d_leaf_rng.p, T.d_blk_off.p, T.d_lu.p, T.d_piv.p, d_info.p);
            else
              lu_panel_kernel<<<L.cnt, kPT, sizeof(double) * (size_t)mr * kSP, st>>>(
                  list, L.k0, T.d_leaf_rng.p, T.d_blk_off.p, T.d_lu.p, T.d_piv.p, d_info.p);
            break;
          }
          case 1: {
            TABI_K(K_LU_STRIP, st);
            lu_strip_kernel<<<L.cnt, kUT, 0, st>>>(B.items.p + L.off, L.k0, T.d_leaf_rng.p,
                                                   T.d_blk_off.p, T.d_lu.p, T.d_piv.p);
            break;
          }
          case 2: {
            TABI_K(K_LU_UPDATE, st);
            lu_gemm_kernel<<<L.cnt, kUT, kGemmSmem, st>>>(B.gitems.p + L.off, L.k0, L.kdepth,
                                                          T.d_leaf_rng.p, T.d_blk_off.p,
                                                          T.d_lu.p);
            break;
          }
          case 3: {
            TABI_K(K_LU_SWAP, st);
            lu_swapmap_kernel<<<L.cnt, 256, 0, st>>>(B.mleaves.p + L.off, L.k0,
                                                     T.d_leaf_rng.p, T.d_piv.p, B.map.p);
            break;
          }
          case 4: {
            TABI_K(K_LU_SWAP, st);
            lu_rowswap_kernel<<<L.cnt, kUT, 0, st>>>(B.ritems.p + L.off, T.d_leaf_rng.p,
                                                     T.d_blk_off.p, B.map.p, T.d_lu.p);
            break;
          }
        }
      }
    };
    if (!grp[0].empty()) run_group(grp[0], H.pc_plan[0], s);
    if (!grp[1].empty()) run_group(grp[1], H.pc_plan[1], split ? H.side : s);
    join(split);
    if (any_big) {
      H.pc_big.alloc(big_leaves.size());
      TABI_CUDA(cudaMemcpyAsync(H.pc_big.p, big_leaves.data(), sizeof(int) * big_leaves.size(),
                                cudaMemcpyHostToDevice, s));
      TABI_K(K_LU, s);
      lu_kernel<<<(int)big_leaves.size(), kLuThreads, 0, s>>>(
          H.pc_big.p, T.d_leaf_rng.p, T.d_blk_off.p, T.d_lu.p, T.d_piv.p, d_info.p, kPanelMaxM);
    }
  // pivot permutations and inverse diagonal blocks for the applies
  {
    T.dinv_off.resize(nl);
    int64_t doff = 0;
    std::vector<int2> dblocks;
    for (int l = 0; l < nl; ++l) {
      T.dinv_off[l] = doff;
      int m = 2 * rng[l].y;
      int nblk = (m + kDB - 1) / kDB;
      doff += (int64_t)nblk * 2 * kDB * kDB;
      for (int b = 0; b < nblk; ++b) dblocks.push_back(make_int2(l, b * kDB));
    }
    while (dblocks.size() % 4) dblocks.push_back(make_int2(-1, 0));
    T.d_dinv.alloc(std::max<int64_t>(doff, 1));
    T.d_dinv_off.alloc(nl);
    T.d_lu_perm.alloc(2 * (size_t)H.n);
    H.pc_dblocks.alloc(std::max<size_t>(dblocks.size(), 1));
    TABI_CUDA(cudaMemcpyAsync(T.d_dinv_off.p, T.dinv_off.data(), sizeof(int64_t) * nl,
                              cudaMemcpyHostToDevice, s));
    TABI_CUDA(cudaMemcpyAsync(H.pc_dblocks.p, dblocks.data(), sizeof(int2) * dblocks.size(),
                              cudaMemcpyHostToDevice, s));
    { TABI_K(K_LU_POST, s); lu_perm_kernel<<<ceil_div(nl, 64), 64, 0, s>>>(T.d_leaf_rng.p, T.d_piv.p, nl, T.d_lu_perm.p); }
    { TABI_K(K_LU_POST, s); lu_diaginv_kernel<<<(int)(dblocks.size() / 4), 128, 0, s>>>(
        H.pc_dblocks.p, T.d_leaf_rng.p, T.d_blk_off.p, T.d_dinv_off.p, T.d_lu.p, T.d_dinv.p,
        d_info.p); }
  }
  }
  {
    std::vector<int> info(nl);
    TABI_CUDA(cudaMemcpyAsync(info.data(), d_info.p, sizeof(int) * nl, cudaMemcpyDeviceToHost,
                              s));
    TABI_CUDA(cudaStreamSynchronize(s));
    for (int l = 0; l < nl; ++l) {
      if (info[l] > 0)
        throw Error(TABI_ERR_SINGULAR, "leaf block " + std::to_string(l) +
                                           " is singular (DGETRF info " +
                                           std::to_string(info[l]) + ")");
      if (info[l] < 0)
        throw Error(TABI_ERR_SINGULAR, "leaf block " + std::to_string(l) +
                                           " has a non-finite pivot at row " +
                                           std::to_string(-info[l]) +
                                           " (coincident faces or non-finite surface data)");
    }
  }
  H.pc_lu_phase.reset();
  H.has_precond = true;
}

void msolve_dev(Handle& H, const double* r, double* z, cudaStream_t s) {
  Tree& T = H.tree;
  const int n = H.n;
  double eps = H.prm.eps1 / H.prm.eps0;
  if (H.prm.iprcd != 1) {
    { TABI_K(K_SOLVE, s); diag_kernel<<<ceil_div(2 * n, 256), 256, 0, s>>>(r, z, n, 0.5 * (1.0 + eps),
                                                     0.5 * (1.0 + 1.0 / eps)); }
    TABI_CUDA(cudaGetLastError());
    return;
  }
  TABI_PHASE(K_PHASE_APPLY, s);
  TABI_REQUIRE(T.max_leaf <= kMaxSolveLeaf, TABI_ERR_LIMIT, "leaf too large for the block solve");
  // a shard applies the leaves of its target range only
  const int nbig = T.ranged ? T.r_solve_big : T.n_solve_big;
  const int nsmall = T.ranged ? T.r_solve_small : T.n_solve_small;
  const int* list = T.ranged ? T.d_r_solve_list.p : T.d_solve_list.p;
  const bool fork = nbig > 0 && nsmall > 0 && H.side != nullptr;
  cudaStream_t s2 = fork ? H.side : s;
  if (fork) {
    TABI_CUDA(cudaEventRecord(H.ev_fork, s));
    TABI_CUDA(cudaStreamWaitEvent(s2, H.ev_fork, 0));
  }
  auto launch = [&](auto* kernel, int threads, size_t smem, int count, const int* leaves,
                    cudaStream_t st) {
    if (count == 0) return;
    raise_smem_limit((const void*)kernel, smem);
    TABI_K(K_SOLVE, st);
    kernel<<<count, threads, smem, st>>>(T.d_leaf_rng.p, T.d_blk_off.p, T.d_dinv_off.p,
                                                  leaves, T.d_lu.p, T.d_dinv.p, T.d_lu_perm.p, n,
                                                  r, z);
  };
  const int order = 2 * T.max_leaf;
  if (T.solve_rows)
    launch(solve_rows_kernel, kRowThreads, row_bytes(order), nbig, list, s);
  else if (order <= kSolveHuge)
    launch(solve_kernel<2, kRingBig>, solve_threads(2), solve_bytes(2, kRingBig, order), nbig,
           list, s);
  else  // the vector (92 KB for the largest leaf) leaves room for fewer tiles
    launch(solve_kernel<2, kRingHuge>, solve_threads(2), solve_bytes(2, kRingHuge, order), nbig,
           list, s);
  launch(solve_kernel<1, kRingSmall>, solve_threads(1),
         solve_bytes(1, kRingSmall, std::min(order, kSolveSmall)), nsmall, list + nbig, s2);
  if (fork) {
    TABI_CUDA(cudaEventRecord(H.ev_join, s2));
    TABI_CUDA(cudaStreamWaitEvent(s, H.ev_join, 0));
  }
  TABI_CUDA(cudaGetLastError());
}

}  // namespace tabi
