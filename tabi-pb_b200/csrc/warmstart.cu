// warmstart.cu -- the learned warm start: a rotation- and translation-invariant
// point-cloud network over surface panels that predicts the initial surface
// potential and normal derivative x0 = [phi; dphi/dn] of a solve from the
// panel geometry and the right-hand side (main.f90:592-606).  It has no
// counterpart in the reference, which always starts GMRES from zero
// (main.f90:133); GMRES on the true residual still decides convergence, so a
// prediction only changes the iteration count.
//
// Network, for N panels (centroid r, unit normal n, area A, b = [b1; b2], and
// z = M^-1 b, the leaf-block preconditioner's solution -- exact within each
// leaf -- or [0; b2] without it):
//   graph   K = 16 nearest other panels per panel (cell-list search, exact,
//           ascending distance, ties by index)
//   input   10 invariant node features (asinh of z / s among them) and 11
//           invariant edge features (8 radial basis functions of |r_ij| /
//           mean neighbour distance and three normal/direction cosines)
//   layers  h = silu(f W0 + b0); L times: u = h Wa,
//           a_i = 1/K sum_k silu(e_ij Wf + bf) * u_j, g = h Wb1 + a Wb2 + bb,
//           h += silu(g)
//   output  o = h Wo + bo, x = z + s o with s = rms(b1): the network corrects z
// Weight matrices are used in bfloat16 with FP32 accumulation; FP32 master
// weights, gradients and Adam moments are kept for training.  Every reduction
// (weight gradients, bias gradients, loss) is a fixed-order two-stage sum, and
// the scatter of the aggregation's backward pass runs as a gather over the
// reversed neighbour lists, so a training step is deterministic.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <type_traits>

#include "tabi_impl.cuh"
#include "warmstart.cuh"

namespace tabi {

namespace {

constexpr int kK = kWsK;      // neighbours
constexpr int kR = kWsR;      // radial basis functions
constexpr int kE = kWsR + 3;  // edge features
constexpr int kF = kWsF;      // node features
constexpr int kRedB = 592;    // blocks of the fixed-grid reductions
constexpr int kWsBlocks = 592;

// 1/(1 + e^-x) with the bits of the IEEE quotient, without the division's branch:
// the hardware's reciprocal (within an ulp) and one multiply-add of its residual,
// which rounds correctly (Markstein, IBM J. Res. Dev. 34 (1990)).  All of it at
// 2^-24 of y = 1 + e^-x, exact until the last product: the approximation flushes a
// subnormal result to zero, and 1/y is one from x = -87.3 on (rounded twice there,
// within 2^-149 of the quotient).  An infinite e^-x gives 0.  The division for
// those y behind a branch instead: 10-15 % on a gradient.
__device__ __forceinline__ float sigm(float x) {
  const float y = fminf(fmaf(__expf(-x), 0x1p-24f, 0x1p-24f), 3e38f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return fmaf(r, fmaf(-y, r, 1.f), r) * 0x1p-24f;
}
__device__ __forceinline__ float silu(float x) { return x * sigm(x); }
__device__ __forceinline__ float dsilu(float x) {
  const float s = sigm(x);
  return s * (1.f + x * (1.f - s));
}

// ---------------------------------------------------------------- inputs
// Panels to FP32 (position + area, normal) from strided FP64 components, and
// per-block partial sums of area, b1^2 and the bounding box.
__global__ void ws_prep_kernel(int n, const double* __restrict__ px, const double* __restrict__ py,
                               const double* __restrict__ pz, int ps,
                               const double* __restrict__ qx, const double* __restrict__ qy,
                               const double* __restrict__ qz, int qs,
                               const double* __restrict__ area, const double* __restrict__ b,
                               const double* __restrict__ zp, float4* __restrict__ pos,
                               float4* __restrict__ nrm, float2* __restrict__ bf,
                               float2* __restrict__ zf, double* __restrict__ part) {
  double sa = 0.0, sb = 0.0;
  float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = px[(size_t)i * ps], y = py[(size_t)i * ps], z = pz[(size_t)i * ps];
    const double a = area[i];
    pos[i] = make_float4((float)x, (float)y, (float)z, (float)a);
    nrm[i] = make_float4((float)qx[(size_t)i * qs], (float)qy[(size_t)i * qs],
                         (float)qz[(size_t)i * qs], 0.f);
    bf[i] = make_float2((float)b[i], (float)b[n + i]);
    zf[i] = zp ? make_float2((float)zp[i], (float)zp[n + i]) : make_float2(0.f, (float)b[n + i]);
    sa += a;
    sb += b[i] * b[i];
    const float c[3] = {(float)x, (float)y, (float)z};
    for (int d = 0; d < 3; ++d) {
      lo[d] = fminf(lo[d], c[d]);
      hi[d] = fmaxf(hi[d], c[d]);
    }
  }
  __shared__ double s[8][256];
  const int t = threadIdx.x;
  s[0][t] = sa;
  s[1][t] = sb;
  for (int d = 0; d < 3; ++d) {
    s[2 + d][t] = lo[d];
    s[5 + d][t] = hi[d];
  }
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (t < w) {
      s[0][t] += s[0][t + w];
      s[1][t] += s[1][t + w];
      for (int d = 0; d < 3; ++d) {
        s[2 + d][t] = fmin(s[2 + d][t], s[2 + d][t + w]);
        s[5 + d][t] = fmax(s[5 + d][t], s[5 + d][t + w]);
      }
    }
    __syncthreads();
  }
  if (t < 8) part[blockIdx.x * 8 + t] = s[t][0];
}

__global__ void ws_prep_final_kernel(const double* __restrict__ part, int nb, double* out) {
  if (threadIdx.x != 0) return;
  double v[8] = {0, 0, 3e38, 3e38, 3e38, -3e38, -3e38, -3e38};
  for (int k = 0; k < nb; ++k) {
    v[0] += part[8 * k];
    v[1] += part[8 * k + 1];
    for (int d = 0; d < 3; ++d) {
      v[2 + d] = fmin(v[2 + d], part[8 * k + 2 + d]);
      v[5 + d] = fmax(v[5 + d], part[8 * k + 5 + d]);
    }
  }
  for (int k = 0; k < 8; ++k) out[k] = v[k];
}

// ---------------------------------------------------------------- graph
struct Grid {
  float x0, y0, z0, h;
  int nx, ny, nz;
};

__device__ __forceinline__ int cell_coord(float v, float v0, float h, int nmax) {
  int c = (int)floorf((v - v0) / h);
  return min(max(c, 0), nmax - 1);
}

__global__ void ws_cell_count_kernel(int n, const float4* __restrict__ pos, Grid g,
                                     int* __restrict__ cell, int* __restrict__ cnt) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 p = pos[i];
  int c = (cell_coord(p.z, g.z0, g.h, g.nz) * g.ny + cell_coord(p.y, g.y0, g.h, g.ny)) * g.nx +
          cell_coord(p.x, g.x0, g.h, g.nx);
  cell[i] = c;
  atomicAdd(&cnt[c], 1);
}

__global__ void ws_cell_fill_kernel(int n, const int* __restrict__ cell,
                                    int* __restrict__ cursor, int* __restrict__ sorted) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  sorted[atomicAdd(&cursor[cell[i]], 1)] = i;
}

// exclusive scan of cnt[0..m) into off[0..m], three passes (block sums,
// scan of the block sums, add)
constexpr int kScanB = 1024;
__global__ void ws_scan_block_kernel(const int* __restrict__ in, int m, int* __restrict__ out,
                                     int* __restrict__ bsum) {
  __shared__ int s[kScanB];
  int i = blockIdx.x * kScanB + threadIdx.x;
  int v = i < m ? in[i] : 0;
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < kScanB; o <<= 1) {
    int t = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
    __syncthreads();
    s[threadIdx.x] += t;
    __syncthreads();
  }
  if (i < m) out[i] = s[threadIdx.x] - v;
  if (threadIdx.x == kScanB - 1) bsum[blockIdx.x] = s[threadIdx.x];
}

__global__ void ws_scan_sums_kernel(int* __restrict__ bsum, int nb, int* __restrict__ total) {
  if (threadIdx.x != 0) return;
  int acc = 0;
  for (int k = 0; k < nb; ++k) {
    int v = bsum[k];
    bsum[k] = acc;
    acc += v;
  }
  *total = acc;
}

__global__ void ws_scan_add_kernel(int* __restrict__ out, int m, const int* __restrict__ bsum,
                                   const int* __restrict__ total) {
  int i = blockIdx.x * kScanB + threadIdx.x;
  if (i < m) out[i] += bsum[blockIdx.x];
  if (i == 0) out[m] = *total;
}

// K nearest other panels: search the cube of cells within +-rad of the
// panel's cell; the result is exact once the K-th distance is within rad*h
// (the cube contains that ball), else the cube grows -- at most until it
// covers the grid (panels of small isolated surface pieces, e.g. cavities of
// fewer than K + 1 faces, find their neighbours on another piece far away).
__global__ void ws_knn_kernel(int n, const float4* __restrict__ pos, Grid g,
                              const int* __restrict__ coff, const int* __restrict__ sorted,
                              int* __restrict__ nbr, int* __restrict__ err) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 p = pos[i];
  const int cx = cell_coord(p.x, g.x0, g.h, g.nx), cy = cell_coord(p.y, g.y0, g.h, g.ny),
            cz = cell_coord(p.z, g.z0, g.h, g.nz);
  float bd[kK];
  int bi[kK];
  // the cube grows by one cell to rad 4, then doubles (isolated pieces)
  for (int rad = 1;; rad = rad < 4 ? rad + 1 : 2 * rad) {
#pragma unroll
    for (int k = 0; k < kK; ++k) {
      bd[k] = 3e38f;
      bi[k] = 0x7fffffff;
    }
    for (int z = max(cz - rad, 0); z <= min(cz + rad, g.nz - 1); ++z)
      for (int y = max(cy - rad, 0); y <= min(cy + rad, g.ny - 1); ++y)
        for (int x = max(cx - rad, 0); x <= min(cx + rad, g.nx - 1); ++x) {
          const int c = (z * g.ny + y) * g.nx + x;
          for (int q = coff[c]; q < coff[c + 1]; ++q) {
            const int j = sorted[q];
            if (j == i) continue;
            const float4 o = pos[j];
            const float dx = o.x - p.x, dy = o.y - p.y, dz = o.z - p.z;
            const float d = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (d > bd[kK - 1] || (d == bd[kK - 1] && j > bi[kK - 1])) continue;
            // insert (d, j) keeping (distance, index) ascending
            float cd = d;
            int cj = j;
#pragma unroll
            for (int k = 0; k < kK; ++k) {
              const bool less = cd < bd[k] || (cd == bd[k] && cj < bi[k]);
              const float td = bd[k];
              const int tj = bi[k];
              bd[k] = less ? cd : td;
              bi[k] = less ? cj : tj;
              cd = less ? td : cd;
              cj = less ? tj : cj;
            }
          }
        }
    const float reach = rad * g.h;
    const bool whole = cx - rad <= 0 && cy - rad <= 0 && cz - rad <= 0 && cx + rad >= g.nx - 1 &&
                       cy + rad >= g.ny - 1 && cz + rad >= g.nz - 1;
    if ((bi[kK - 1] != 0x7fffffff && bd[kK - 1] <= reach * reach) || whole) break;
  }
  // fewer than K other panels exist only when n <= K, which the host rejects
  if (bi[kK - 1] == 0x7fffffff) atomicExch(err, 1);
#pragma unroll
  for (int k = 0; k < kK; ++k) nbr[(size_t)i * kK + k] = bi[k] == 0x7fffffff ? i : bi[k];
}

// reversed neighbour lists: for panel j, the edges (i, k) with nbr(i, k) = j
__global__ void ws_rev_count_kernel(int n, const int* __restrict__ nbr, int* __restrict__ cnt) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * kK) return;
  atomicAdd(&cnt[nbr[e]], 1);
}

__global__ void ws_rev_fill_kernel(int n, const int* __restrict__ nbr, int* __restrict__ cursor,
                                   int* __restrict__ rev) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * kK) return;
  rev[atomicAdd(&cursor[nbr[e]], 1)] = e;
}

// each list in ascending edge id (fixed order for the gather)
__global__ void ws_rev_sort_kernel(int n, const int* __restrict__ off, int* __restrict__ rev) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int a = off[j], b = off[j + 1];
  for (int p = a + 1; p < b; ++p) {
    int v = rev[p], q = p - 1;
    while (q >= a && rev[q] > v) {
      rev[q + 1] = rev[q];
      --q;
    }
    rev[q + 1] = v;
  }
}

// edge features e_ij (kE) of panel i's neighbour j
__device__ __forceinline__ void edge_feat(const float4 pi, const float4 ni, const float4 pj,
                                          const float4 nj, float dbar, float* e) {
  const float rx = pj.x - pi.x, ry = pj.y - pi.y, rz = pj.z - pi.z;
  const float d = sqrtf(fmaf(rx, rx, fmaf(ry, ry, rz * rz)));
  const float inv = d > 0.f ? 1.f / d : 0.f;
  const float rho = d / dbar;
  const float sig = 2.5f / (kR - 1);
#pragma unroll
  for (int m = 0; m < kR; ++m) {
    const float t = (rho - sig * m) / sig;
    e[m] = __expf(-t * t);
  }
  e[kR] = fmaf(ni.x, nj.x, fmaf(ni.y, nj.y, ni.z * nj.z));
  e[kR + 1] = fmaf(ni.x, rx, fmaf(ni.y, ry, ni.z * rz)) * inv;
  e[kR + 2] = fmaf(nj.x, rx, fmaf(nj.y, ry, nj.z * rz)) * inv;
}

// node features (kF per panel) and the mean neighbour distance
__global__ void ws_node_kernel(int n, const float4* __restrict__ pos, const float4* __restrict__ nrm,
                               const float2* __restrict__ bf, const float2* __restrict__ zf,
                               const int* __restrict__ nbr,
                               const double* __restrict__ stats, float* __restrict__ dbar_out,
                               float* __restrict__ f) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float abar = (float)(stats[0] / n);
  double ms = stats[1] / n;
  const float s = ms > 0.0 ? (float)sqrt(ms) : 1.f;
  const float4 p = pos[i], q = nrm[i];
  const float2 bi = bf[i];
  float dsum = 0.f, curv = 0.f, nn = 0.f, db = 0.f;
  float dd[kK], hh[kK];
#pragma unroll
  for (int k = 0; k < kK; ++k) {
    const int j = nbr[(size_t)i * kK + k];
    const float4 o = pos[j], m = nrm[j];
    const float rx = o.x - p.x, ry = o.y - p.y, rz = o.z - p.z;
    const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
    dd[k] = d2;
    hh[k] = fmaf(q.x, rx, fmaf(q.y, ry, q.z * rz));
    dsum += sqrtf(d2);
    nn += fmaf(q.x, m.x, fmaf(q.y, m.y, q.z * m.z));
    db += (bf[j].x - bi.x) / s;
  }
  const float dbar = fmaxf(dsum / kK, 1e-6f);
#pragma unroll
  for (int k = 0; k < kK; ++k) curv += dd[k] > 0.f ? hh[k] * dbar / dd[k] : 0.f;
  dbar_out[i] = dbar;
  float* o = f + (size_t)i * kF;
  o[0] = bi.x / s;
  o[1] = bi.y / s;
  o[2] = logf(fmaxf(p.w / abar, 1e-6f));
  o[3] = logf(abar);
  o[4] = curv / kK;
  o[5] = nn / kK;
  o[6] = logf(dbar);
  o[7] = db / kK;
  const float2 zi = zf[i];
  // z can be far off on poorly conditioned molecules: asinh keeps the input
  // bounded (linear near zero, logarithmic beyond)
  o[8] = asinhf(zi.x / s);
  o[9] = asinhf((zi.y - bi.y) / s);
}

// ---------------------------------------------------------------- dense layers
// C (M x N) = A (M x Kd, FP32, row-major) * B, B in bfloat16: B(k, c) = W[k*ldw + c]
// (TB = false) or W[c*ldw + k] (TB = true, i.e. A * W^T).  Epilogues:
//   0: C = acc            1: C = acc + bias          2: C += acc
//   3: P = acc + bias, C = silu(P)
//   4: P = P_in + acc, C = R + silu(P)  (second half of z = h Wb1 + a Wb2 + bb,
//      P_in = h Wb1 + bb; R the residual input h)
// A block takes 64 rows and 16 T columns -- all of them up to a width of 160, where
// there are rows enough -- in 16-deep k steps, 4 x T outputs per thread (one 16-byte and T/2 8-byte shared
// loads for 4 T multiply-adds), the next step's operands in registers
// meanwhile; three blocks per SM where the epilogue reads two more matrices,
// else two with the accumulators' registers unspilled.  Each output is one
// chain of multiply-adds in order of k, so the tile shape does not change it.
// Bound by issue and shared loads.  77,594 x 160 x 160, A W: 160 -> 129 us, with
// epilogue 4 197 -> 195; the 64 x 64 tiles of 4 x 4 outputs wasted a sixth of
// their columns and waited for every step's loads.
constexpr int kGM = 64, kGK = 16;

template <int T, bool TB, int EPI>
__global__ void __launch_bounds__(256, EPI <= 1 ? 2 : 3) ws_gemm_kernel(int M, int N, int Kd,
                                                      const float* __restrict__ A, int lda,
                                                      const __nv_bfloat16* __restrict__ W,
                                                      int ldw, const float* __restrict__ bias,
                                                      float* __restrict__ C, int ldc,
                                                      float* __restrict__ P,
                                                      const float* __restrict__ Rin) {
  constexpr int BN = 16 * T;
  __shared__ __align__(16) float As[kGK][kGM + 4];
  __shared__ __align__(8) float Bs[kGK][BN + 2];
  const int tid = threadIdx.x;
  const int tr = tid / 16, tc = tid % 16;
  const int row0 = blockIdx.x * kGM, col0 = blockIdx.y * BN;
  const int ar = tid / 4, ak = 4 * (tid % 4);  // this thread's 4 elements of an A step
  float av[4];
  __nv_bfloat16 bv[T];
  auto fetch = [&](int k0) {
    const int gr = row0 + ar;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      av[q] = gr < M && k0 + ak + q < Kd ? A[(size_t)gr * lda + k0 + ak + q] : 0.f;
#pragma unroll
    for (int q = 0; q < T; ++q) {
      const int e = tid + q * 256;
      const int bk = TB ? e % kGK : e / BN, bc = TB ? e / kGK : e % BN;
      const int gk = k0 + bk, gc = col0 + bc;
      bv[q] = gk < Kd && gc < N ? (TB ? W[(size_t)gc * ldw + gk] : W[(size_t)gk * ldw + gc])
                                : __float2bfloat16(0.f);
    }
  };
  float acc[4][T] = {};
  fetch(0);
  for (int k0 = 0; k0 < Kd; k0 += kGK) {
    if (k0 > 0) __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) As[ak + q][ar] = av[q];
#pragma unroll
    for (int q = 0; q < T; ++q) {
      const int e = tid + q * 256;
      Bs[TB ? e % kGK : e / BN][TB ? e / kGK : e % BN] = __bfloat162float(bv[q]);
    }
    __syncthreads();
    if (k0 + kGK < Kd) fetch(k0 + kGK);
#pragma unroll
    for (int k = 0; k < kGK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&As[k][tr * 4]);
      float b[T];
#pragma unroll
      for (int j = 0; j < T; j += 2) {
        if (j + 1 < T) {
          const float2 v = *reinterpret_cast<const float2*>(&Bs[k][2 * tc + 16 * j]);
          b[j] = v.x;
          b[j + 1] = v.y;
        } else {
          b[j] = Bs[k][tc + 16 * j];
        }
      }
#pragma unroll
      for (int j = 0; j < T; ++j) {
        acc[0][j] = fmaf(a.x, b[j], acc[0][j]);
        acc[1][j] = fmaf(a.y, b[j], acc[1][j]);
        acc[2][j] = fmaf(a.z, b[j], acc[2][j]);
        acc[3][j] = fmaf(a.w, b[j], acc[3][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = row0 + tr * 4 + i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < T; ++j) {
      // columns in pairs (the last of an odd T alone), as they were read
      const int c = col0 + (j + 1 < T || (j & 1) ? 2 * tc + 16 * (j & ~1) + (j & 1) : tc + 16 * j);
      if (c >= N) continue;
      const size_t o = (size_t)r * ldc + c;
      const float v = acc[i][j];
      if (EPI == 0) C[o] = v;
      if (EPI == 1) C[o] = v + bias[c];
      if (EPI == 2) C[o] += v;
      if (EPI == 3) {
        const float pr = v + bias[c];
        P[o] = pr;
        C[o] = silu(pr);
      }
      if (EPI == 4) {
        const float pr = P[o] + v;
        P[o] = pr;
        C[o] = Rin[o] + silu(pr);
      }
    }
  }
}

// Weight gradient partials: part[chunk] (Kd x N) = A[rows of chunk]^T * D[rows of
// chunk].  A block takes 16 T x 16 T outputs, T x T per thread (T 8-byte shared
// loads for T^2 multiply-adds); the chunks are short enough to give every SM two
// blocks.  77,594 rows, 160 x 160: 583 us with 64 x 64 tiles over 4,096 rows (171
// blocks of 4 x 4 outputs per thread) -> 101 us.
template <int T>
__global__ void __launch_bounds__(256) ws_dw_kernel(int M, int Kd, int N, int chunk,
                                                    const float* __restrict__ A, int lda,
                                                    const float* __restrict__ D, int ldd,
                                                    float* __restrict__ part) {
  constexpr int BT = 16 * T;
  __shared__ __align__(8) float As[kGK][BT], Ds[kGK][BT];
  // outputs in pairs (the last of an odd T alone)
  auto at = [](int t, int q) {
    return q + 1 < T || (q & 1) ? 2 * t + 16 * (q & ~1) + (q & 1) : t + 16 * q;
  };
  const int tid = threadIdx.x;
  const int tr = tid / 16, tc = tid % 16;
  const int k0 = blockIdx.x * BT, c0 = blockIdx.y * BT;
  const int m0 = blockIdx.z * chunk, m1 = min(M, m0 + chunk);
  float av[T], dv[T];
  auto fetch = [&](int mb) {
#pragma unroll
    for (int q = 0; q < T; ++q) {
      const int e = tid + q * 256, r = e / BT, c = e % BT, gm = mb + r;
      av[q] = gm < m1 && k0 + c < Kd ? A[(size_t)gm * lda + k0 + c] : 0.f;
      dv[q] = gm < m1 && c0 + c < N ? D[(size_t)gm * ldd + c0 + c] : 0.f;
    }
  };
  float acc[T][T] = {};
  fetch(m0);
  for (int mb = m0; mb < m1; mb += kGK) {
    if (mb > m0) __syncthreads();
#pragma unroll
    for (int q = 0; q < T; ++q) {
      const int e = tid + q * 256;
      As[e / BT][e % BT] = av[q];
      Ds[e / BT][e % BT] = dv[q];
    }
    __syncthreads();
    if (mb + kGK < m1) fetch(mb + kGK);
#pragma unroll 4
    for (int r = 0; r < kGK; ++r) {
      float a[T], d[T];
#pragma unroll
      for (int i = 0; i < T; i += 2) {
        if (i + 1 < T) {
          const float2 v = *reinterpret_cast<const float2*>(&As[r][at(tr, i)]);
          const float2 w = *reinterpret_cast<const float2*>(&Ds[r][at(tc, i)]);
          a[i] = v.x;
          a[i + 1] = v.y;
          d[i] = w.x;
          d[i + 1] = w.y;
        } else {
          a[i] = As[r][at(tr, i)];
          d[i] = Ds[r][at(tc, i)];
        }
      }
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) acc[i][j] = fmaf(a[i], d[j], acc[i][j]);
    }
  }
  float* out = part + (size_t)blockIdx.z * Kd * N;
#pragma unroll
  for (int i = 0; i < T; ++i) {
    const int k = k0 + at(tr, i);
    if (k >= Kd) continue;
#pragma unroll
    for (int j = 0; j < T; ++j) {
      const int c = c0 + at(tc, j);
      if (c < N) out[(size_t)k * N + c] = acc[i][j];
    }
  }
}

// g[e] = sum over chunks of part[chunk][e]: 32 elements per block, 8 threads
// each over every 8th chunk in order, their sums added in order in FP64
__global__ void __launch_bounds__(256) ws_sum_parts_kernel(const float* __restrict__ part,
                                                           int nchunk, int64_t len,
                                                           float* __restrict__ g) {
  __shared__ double sm[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t e = blockIdx.x * (int64_t)32 + lane;
  double s = 0.0;
  if (e < len)
#pragma unroll 4
    for (int c = w; c < nchunk; c += 8) s += part[(size_t)c * len + e];
  sm[w][lane] = s;
  __syncthreads();
  if (w == 0 && e < len) {
#pragma unroll
    for (int q = 1; q < 8; ++q) s += sm[q][lane];
    g[e] = (float)s;
  }
}

// column sums of X (M x N) into part[block][N] (fixed row ranges per block)
__global__ void ws_colsum_kernel(int M, int N, const float* __restrict__ X,
                                 float* __restrict__ part) {
  const int per = (M + gridDim.x - 1) / gridDim.x;
  const int r0 = blockIdx.x * per, r1 = min(M, r0 + per);
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    float s = 0.f;
    for (int r = r0; r < r1; ++r) s += X[(size_t)r * N + c];
    part[(size_t)blockIdx.x * N + c] = s;
  }
}

// elementwise: out = g * silu'(x)
__global__ void ws_dsilu_kernel(int64_t len, const float* __restrict__ g,
                                const float* __restrict__ x, float* __restrict__ out) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len;
       e += (int64_t)gridDim.x * blockDim.x)
    out[e] = g[e] * dsilu(x[e]);
}

// ---------------------------------------------------------------- aggregation
// a_i = 1/K sum_k silu(e_ik Wf + bf) * u_{nbr(i,k)}.  A block of H threads takes
// kGrp panels at a time, H/4 threads per panel and 4 channels per thread: an
// edge's 12 padded features are three 16-byte shared loads for 44
// multiply-adds, and the neighbour's channels one 16-byte load (one channel
// per thread read 11 words for 11 multiply-adds).  Every panel's sums run in
// the order of its edges.  Bound by the latency of the gate's exponential and
// reciprocal.  77,594 panels, H = 160: 400 -> 242 us.
constexpr int kGrp = 4;
constexpr int kWsNodes = 16;  // panels per block of the forward and du kernels

struct EdgeStage {
  float4 e[kGrp][kK][3];
  int j[kGrp][kK];
};

// the weights of 4 channels
struct Chan4 {
  float4 w[kE], b;
  __device__ __forceinline__ void load(const __nv_bfloat16* Wf, const float* bf, int H, int c) {
#pragma unroll
    for (int q = 0; q < kE; ++q) {
      const __nv_bfloat16* p = Wf + (size_t)q * H + c;
      w[q] = make_float4(__bfloat162float(p[0]), __bfloat162float(p[1]), __bfloat162float(p[2]),
                         __bfloat162float(p[3]));
    }
    b = make_float4(bf[c], bf[c + 1], bf[c + 2], bf[c + 3]);
  }
  __device__ __forceinline__ float4 pre(const float (&e)[12]) const {
    float4 v = b;
#pragma unroll
    for (int q = 0; q < kE; ++q) {
      v.x = fmaf(e[q], w[q].x, v.x);
      v.y = fmaf(e[q], w[q].y, v.y);
      v.z = fmaf(e[q], w[q].z, v.z);
      v.w = fmaf(e[q], w[q].w, v.w);
    }
    return v;
  }
};

__device__ __forceinline__ void edge_unpack(const float4 (&s)[3], float (&e)[12]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float4 v = s[q];
    e[4 * q] = v.x;
    e[4 * q + 1] = v.y;
    e[4 * q + 2] = v.z;
    e[4 * q + 3] = v.w;
  }
}

__device__ __forceinline__ void edge_stage(float4 (&dst)[3], const float4 pi, const float4 ni,
                                           const float4 pj, const float4 nj, float dbar) {
  static_assert(kE <= 12, "an edge's features are three float4");
  float e[12] = {};
  float f[kE];
  edge_feat(pi, ni, pj, nj, dbar, f);
#pragma unroll
  for (int q = 0; q < kE; ++q) e[q] = f[q];
#pragma unroll
  for (int q = 0; q < 3; ++q)
    dst[q] = make_float4(e[4 * q], e[4 * q + 1], e[4 * q + 2], e[4 * q + 3]);
}

// the edges of panels i0 .. i0 + kGrp (below iend) into shared memory
__device__ __forceinline__ void stage_panels(EdgeStage& S, int i0, int iend, const float4* pos,
                                             const float4* nrm, const float* dbar,
                                             const int* nbr) {
  for (int q = threadIdx.x; q < kGrp * kK; q += blockDim.x) {
    const int g = q / kK, k = q % kK, i = i0 + g;
    if (i >= iend) continue;
    const int j = nbr[(size_t)i * kK + k];
    S.j[g][k] = j;
    edge_stage(S.e[g][k], pos[i], nrm[i], pos[j], nrm[j], dbar[i]);
  }
}

__global__ void __launch_bounds__(256, 3) ws_agg_fwd_kernel(int n, int H, const float4* __restrict__ pos,
                                  const float4* __restrict__ nrm, const float* __restrict__ dbar,
                                  const int* __restrict__ nbr,
                                  const __nv_bfloat16* __restrict__ Wf,
                                  const float* __restrict__ bfv, const float* __restrict__ u,
                                  float* __restrict__ a) {
  __shared__ EdgeStage S;
  const int g = threadIdx.x / (H / 4), c = 4 * (threadIdx.x % (H / 4));
  Chan4 ch;
  ch.load(Wf, bfv, H, c);
  for (int t = 0; t < kWsNodes; t += kGrp) {
    const int i0 = blockIdx.x * kWsNodes + t, i = i0 + g;
    if (i0 >= n) break;
    __syncthreads();
    stage_panels(S, i0, n, pos, nrm, dbar, nbr);
    __syncthreads();
    if (i >= n) continue;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < kK; ++k) {
      float e[12];
      edge_unpack(S.e[g][k], e);
      const float4 uj = *reinterpret_cast<const float4*>(u + (size_t)S.j[g][k] * H + c);
      const float4 pr = ch.pre(e);
      acc.x = fmaf(silu(pr.x), uj.x, acc.x);
      acc.y = fmaf(silu(pr.y), uj.y, acc.y);
      acc.z = fmaf(silu(pr.z), uj.z, acc.z);
      acc.w = fmaf(silu(pr.w), uj.w, acc.w);
    }
    const float f = 1.f / kK;
    *reinterpret_cast<float4*>(a + (size_t)i * H + c) =
        make_float4(acc.x * f, acc.y * f, acc.z * f, acc.w * f);
  }
}

// Backward of the aggregation, part 1 (contiguous panel ranges per block):
// dpre_ik = u_j da_i / K * silu'(pre_ik); per-block partial gradients of Wf
// (kE x H) and bf (H), the block's groups added in order.  77,594 panels, H = 160:
// 739 -> 450 us.
__global__ void __launch_bounds__(256) ws_agg_bwd_w_kernel(
    int n, int H, const float4* __restrict__ pos, const float4* __restrict__ nrm,
    const float* __restrict__ dbar, const int* __restrict__ nbr,
    const __nv_bfloat16* __restrict__ Wf, const float* __restrict__ bfv,
    const float* __restrict__ u, const float* __restrict__ da, float* __restrict__ part) {
  __shared__ EdgeStage S;
  __shared__ __align__(16) float red[kGrp][256];
  const int g = threadIdx.x / (H / 4), c = 4 * (threadIdx.x % (H / 4));
  Chan4 ch;
  ch.load(Wf, bfv, H, c);
  float4 gw[kE + 1];
#pragma unroll
  for (int q = 0; q <= kE; ++q) gw[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int per = (n + gridDim.x - 1) / gridDim.x;
  const int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
  for (int i0 = b0; i0 < b1; i0 += kGrp) {
    const int i = i0 + g;
    __syncthreads();
    stage_panels(S, i0, b1, pos, nrm, dbar, nbr);
    __syncthreads();
    if (i >= b1) continue;
    float4 d = *reinterpret_cast<const float4*>(da + (size_t)i * H + c);
    const float f = 1.f / kK;
    d = make_float4(d.x * f, d.y * f, d.z * f, d.w * f);
#pragma unroll 2
    for (int k = 0; k < kK; ++k) {
      float e[12];
      edge_unpack(S.e[g][k], e);
      const float4 uj = *reinterpret_cast<const float4*>(u + (size_t)S.j[g][k] * H + c);
      const float4 pr = ch.pre(e);
      const float4 dp = make_float4(uj.x * d.x * dsilu(pr.x), uj.y * d.y * dsilu(pr.y),
                                    uj.z * d.z * dsilu(pr.z), uj.w * d.w * dsilu(pr.w));
#pragma unroll
      for (int q = 0; q < kE; ++q) {
        gw[q].x = fmaf(e[q], dp.x, gw[q].x);
        gw[q].y = fmaf(e[q], dp.y, gw[q].y);
        gw[q].z = fmaf(e[q], dp.z, gw[q].z);
        gw[q].w = fmaf(e[q], dp.w, gw[q].w);
      }
      gw[kE].x += dp.x;
      gw[kE].y += dp.y;
      gw[kE].z += dp.z;
      gw[kE].w += dp.w;
    }
  }
  float* o = part + (size_t)blockIdx.x * (kE + 1) * H;
#pragma unroll
  for (int q = 0; q <= kE; ++q) {
    __syncthreads();
    *reinterpret_cast<float4*>(&red[g][c]) = gw[q];
    __syncthreads();
    float v = red[0][threadIdx.x];
#pragma unroll
    for (int k = 1; k < kGrp; ++k) v += red[k][threadIdx.x];
    o[(size_t)q * H + threadIdx.x] = v;
  }
}

// Backward of the aggregation, part 2 (per panel j, over the reversed lists):
// du_j = sum_{(i,k): nbr(i,k) = j} silu(pre_ik) da_i / K, kK edges of each of the
// block's panels at a time.  77,594 panels, H = 160: 414 -> 322 us.
__global__ void __launch_bounds__(256, 3) ws_agg_bwd_u_kernel(int n, int H, const float4* __restrict__ pos,
                                    const float4* __restrict__ nrm,
                                    const float* __restrict__ dbar, const int* __restrict__ roff,
                                    const int* __restrict__ rev,
                                    const __nv_bfloat16* __restrict__ Wf,
                                    const float* __restrict__ bfv, const float* __restrict__ da,
                                    float* __restrict__ du) {
  __shared__ EdgeStage S;
  const int g = threadIdx.x / (H / 4), c = 4 * (threadIdx.x % (H / 4));
  Chan4 ch;
  ch.load(Wf, bfv, H, c);
  for (int t = 0; t < kWsNodes; t += kGrp) {
    const int j0 = blockIdx.x * kWsNodes + t, j = j0 + g;
    if (j0 >= n) break;
    const int a0 = j < n ? roff[j] : 0, a1 = j < n ? roff[j + 1] : 0;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int b = 0; __syncthreads_or(a0 + b < a1); b += kK) {
      for (int q = threadIdx.x; q < kGrp * kK; q += blockDim.x) {
        const int gg = q / kK, k = q % kK, jj = j0 + gg;
        if (jj >= n) continue;
        const int p = roff[jj] + b + k;
        if (p >= roff[jj + 1]) continue;
        const int i = rev[p] / kK;
        S.j[gg][k] = i;
        edge_stage(S.e[gg][k], pos[i], nrm[i], pos[jj], nrm[jj], dbar[i]);
      }
      __syncthreads();
      const int cnt = min(kK, a1 - a0 - b);
#pragma unroll 4
      for (int k = 0; k < cnt; ++k) {
        float e[12];
        edge_unpack(S.e[g][k], e);
        const float4 d = *reinterpret_cast<const float4*>(da + (size_t)S.j[g][k] * H + c);
        const float4 pr = ch.pre(e);
        acc.x = fmaf(silu(pr.x), d.x, acc.x);
        acc.y = fmaf(silu(pr.y), d.y, acc.y);
        acc.z = fmaf(silu(pr.z), d.z, acc.z);
        acc.w = fmaf(silu(pr.w), d.w, acc.w);
      }
    }
    const float f = 1.f / kK;
    if (j < n)
      *reinterpret_cast<float4*>(du + (size_t)j * H + c) =
          make_float4(acc.x * f, acc.y * f, acc.z * f, acc.w * f);
  }
}

// ---------------------------------------------------------------- head / loss
// o = h Wo + bo (one warp per panel); x = z + s o (z = [0; b2] without a
// preconditioner solution); with a target, do = 2 (o - (x_t - z)/s) / N and
// per-block loss partials.
__global__ void ws_head_kernel(int n, int H, const float* __restrict__ h,
                               const __nv_bfloat16* __restrict__ Wo,
                               const float* __restrict__ bo, const double* __restrict__ b,
                               const double* __restrict__ zp,
                               const double* __restrict__ stats, double* __restrict__ xout,
                               const double* __restrict__ target, float* __restrict__ dout,
                               double* __restrict__ lpart) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double ms = stats[1] / n;
  const double s = ms > 0.0 ? sqrt(ms) : 1.0;
  double lsum = 0.0;
  const int per = (n + gridDim.x - 1) / gridDim.x;
  const int i0 = blockIdx.x * per, i1 = min(n, i0 + per);
  for (int i = i0 + warp; i < i1; i += blockDim.x / 32) {
    float o0 = 0.f, o1 = 0.f;
    for (int c = lane; c < H; c += 32) {
      const float v = h[(size_t)i * H + c];
      o0 = fmaf(v, __bfloat162float(Wo[2 * c]), o0);
      o1 = fmaf(v, __bfloat162float(Wo[2 * c + 1]), o1);
    }
    for (int off = 16; off > 0; off >>= 1) {
      o0 += __shfl_xor_sync(0xffffffffu, o0, off);
      o1 += __shfl_xor_sync(0xffffffffu, o1, off);
    }
    o0 += bo[0];
    o1 += bo[1];
    if (lane == 0) {
      const double z1 = zp ? zp[i] : 0.0, z2 = zp ? zp[n + i] : b[n + i];
      if (xout) {
        xout[i] = z1 + s * o0;
        xout[n + i] = z2 + s * o1;
      }
      if (target) {
        const double t0 = (target[i] - z1) / s, t1 = (target[n + i] - z2) / s;
        const double d0 = o0 - t0, d1 = o1 - t1;
        lsum += d0 * d0 + d1 * d1;
        dout[2 * i] = (float)(2.0 * d0 / n);
        dout[2 * i + 1] = (float)(2.0 * d1 / n);
      }
    }
  }
  if (!target) return;
  __shared__ double sl[32];
  if (lane == 0) sl[warp] = lsum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) t += sl[w];
    lpart[blockIdx.x] = t;
  }
}

__global__ void ws_loss_final_kernel(const double* __restrict__ lpart, int nb, int n,
                                     double* __restrict__ out) {
  if (threadIdx.x != 0) return;
  double t = 0.0;
  for (int k = 0; k < nb; ++k) t += lpart[k];
  out[0] = t / n;
}

// dh = do Wo^T (N x H)
__global__ void ws_head_bwd_kernel(int n, int H, const float* __restrict__ dout,
                                   const __nv_bfloat16* __restrict__ Wo, float* __restrict__ dh) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)n * H;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / H), c = (int)(e % H);
    dh[e] = dout[2 * i] * __bfloat162float(Wo[2 * c]) +
            dout[2 * i + 1] * __bfloat162float(Wo[2 * c + 1]);
  }
}

// ---------------------------------------------------------------- optimiser
__global__ void ws_adam_kernel(int64_t np, float* __restrict__ theta, const float* __restrict__ g,
                               float* __restrict__ m, float* __restrict__ v, float lr, float b1,
                               float b2, float c1, float c2, float eps,
                               __nv_bfloat16* __restrict__ wbf) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < np;
       e += (int64_t)gridDim.x * blockDim.x) {
    const float gv = g[e];
    const float mv = b1 * m[e] + (1.f - b1) * gv;
    const float vv = b2 * v[e] + (1.f - b2) * gv * gv;
    m[e] = mv;
    v[e] = vv;
    const float t = theta[e] - lr * (mv / c1) / (sqrtf(vv / c2) + eps);
    theta[e] = t;
    wbf[e] = __float2bfloat16_rn(t);
  }
}

__global__ void ws_to_bf16_kernel(int64_t np, const float* __restrict__ theta,
                                  __nv_bfloat16* __restrict__ wbf) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < np;
       e += (int64_t)gridDim.x * blockDim.x)
    wbf[e] = __float2bfloat16_rn(theta[e]);
}

void sum_parts(const float* part, int nchunk, int64_t len, float* g, cudaStream_t s) {
  ws_sum_parts_kernel<<<ceil_div(len, 32), 256, 0, s>>>(part, nchunk, len, g);
}

// Column blocks of 16 T for a width N that is a multiple of 32: one up to 160,
// two above; f gets T as a compile-time constant.
template <typename F>
void with_tile(int N, F&& f) {
  switch (N <= 160 ? N / 16 : N / 32) {
    case 2: f(std::integral_constant<int, 2>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    default: f(std::integral_constant<int, 10>()); break;
  }
}

template <bool TB, int EPI>
void gemm(int M, int N, int Kd, const float* A, int lda, const __nv_bfloat16* W, int ldw,
          const float* bias, float* C, int ldc, float* P, const float* R, cudaStream_t s) {
  // the widest column blocks whose grid gives every SM one: all columns from 148
  // blocks of rows on, 64 from 37, else 32 (a prediction at H = 160: 1,112 panels 637,
  // 528 and 511 us, 5,436 panels 696, 636 and 639; 597 and 689 with 64 x 64 tiles)
  const int rows = ceil_div(M, kGM);
  with_tile(rows >= kSMs ? N : rows >= kSMs / 4 ? std::min(N, 64) : 32, [&](auto t) {
    constexpr int T = decltype(t)::value;
    dim3 grid(ceil_div(M, kGM), ceil_div(N, 16 * T));
    ws_gemm_kernel<T, TB, EPI><<<grid, 256, 0, s>>>(M, N, Kd, A, lda, W, ldw, bias, C, ldc, P,
                                                    R);
  });
}

}  // namespace

// ---------------------------------------------------------------- host side
WsNet::WsNet(int hidden, int layers, unsigned long long seed) : H(hidden), L(layers) {
  TABI_REQUIRE(H >= 32 && H <= 256 && H % 32 == 0, TABI_ERR_ARG,
               "hidden width must be a multiple of 32 in 32..256");
  TABI_REQUIRE(L >= 1 && L <= 8, TABI_ERR_ARG, "layers must be in 1..8");
  // flat layout: W0 b0 | per layer Wa Wf bf Wb1 Wb2 bb | Wo bo
  int64_t o = 0;
  auto take = [&](int64_t k) {
    int64_t r = o;
    o += k;
    return r;
  };
  off_W0 = take((int64_t)kF * H);
  off_b0 = take(H);
  for (int l = 0; l < L; ++l) {
    Layer y;
    y.Wa = take((int64_t)H * H);
    y.Wf = take((int64_t)kE * H);
    y.bf = take(H);
    y.Wb1 = take((int64_t)H * H);
    y.Wb2 = take((int64_t)H * H);
    y.bb = take(H);
    lay.push_back(y);
  }
  off_Wo = take((int64_t)H * 2);
  off_bo = take(2);
  np = o;
  // initial weights: N(0, 1/fan_in) for the matrices (the output layer zero,
  // so an untrained network predicts x = z), zero biases
  std::vector<float> th((size_t)np, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<double> nd(0.0, 1.0);
  auto fill = [&](int64_t at, int rows, int cols, double scale) {
    for (int64_t k = 0; k < (int64_t)rows * cols; ++k) th[at + k] = (float)(nd(rng) * scale);
  };
  fill(off_W0, kF, H, 1.0 / std::sqrt((double)kF));
  for (auto& y : lay) {
    fill(y.Wa, H, H, 1.0 / std::sqrt((double)H));
    fill(y.Wf, kE, H, 1.0 / std::sqrt((double)kE));
    fill(y.Wb1, H, H, 0.5 / std::sqrt((double)H));
    fill(y.Wb2, H, H, 0.5 / std::sqrt((double)H));
  }
  TABI_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  h_blk = MemPool::get(sizeof(double) * 16, true);
  h_stats = static_cast<double*>(h_blk.p);
  theta.alloc(np);
  wbf.alloc(np);
  grad.alloc(np);
  m.alloc(np);
  v.alloc(np);
  TABI_CUDA(cudaMemcpyAsync(theta.p, th.data(), sizeof(float) * np, cudaMemcpyHostToDevice,
                            stream));
  TABI_CUDA(cudaMemsetAsync(m.p, 0, sizeof(float) * np, stream));
  TABI_CUDA(cudaMemsetAsync(v.p, 0, sizeof(float) * np, stream));
  ws_to_bf16_kernel<<<256, 256, 0, stream>>>(np, theta.p, wbf.p);
  TABI_CUDA(cudaGetLastError());
  TABI_CUDA(cudaStreamSynchronize(stream));
}

WsNet::~WsNet() {
  if (stream) {
    cudaStreamSynchronize(stream);
    cudaStreamDestroy(stream);
  }
  MemPool::put(h_blk);
}

std::unique_ptr<WsNet> WsNet::clone() const {
  auto c = std::make_unique<WsNet>(H, L, 0ULL);
  TABI_CUDA(cudaMemcpyAsync(c->theta.p, theta.p, sizeof(float) * np, cudaMemcpyDeviceToDevice,
                            c->stream));
  ws_to_bf16_kernel<<<256, 256, 0, c->stream>>>(np, c->theta.p, c->wbf.p);
  TABI_CUDA(cudaGetLastError());
  TABI_CUDA(cudaStreamSynchronize(c->stream));
  return c;
}

void WsNet::set_params(const float* th) {
  TABI_CUDA(cudaMemcpyAsync(theta.p, th, sizeof(float) * np, cudaMemcpyHostToDevice, stream));
  ws_to_bf16_kernel<<<256, 256, 0, stream>>>(np, theta.p, wbf.p);
  TABI_CUDA(cudaGetLastError());
  adam_t = 0;
  TABI_CUDA(cudaMemsetAsync(m.p, 0, sizeof(float) * np, stream));
  TABI_CUDA(cudaMemsetAsync(v.p, 0, sizeof(float) * np, stream));
  TABI_CUDA(cudaStreamSynchronize(stream));
}

void WsNet::get_params(float* th) {
  TABI_CUDA(cudaMemcpyAsync(th, theta.p, sizeof(float) * np, cudaMemcpyDeviceToHost, stream));
  TABI_CUDA(cudaStreamSynchronize(stream));
}

void WsNet::graph(const WsInput& in, cudaStream_t s) {
  const int n = in.n;
  TABI_REQUIRE(n > kK, TABI_ERR_ARG, "the warm start needs more than 16 panels");
  pos.alloc(n);
  nrm.alloc(n);
  bfl.alloc(n);
  zfl.alloc(n);
  const int pb = 148;
  stats_part.alloc(8 * pb + 8);
  stats.alloc(16);
  ws_prep_kernel<<<pb, 256, 0, s>>>(n, in.px, in.py, in.pz, in.ps, in.qx, in.qy, in.qz, in.qs,
                                     in.area, in.b, in.z, pos.p, nrm.p, bfl.p, zfl.p,
                                     stats_part.p);
  ws_prep_final_kernel<<<1, 32, 0, s>>>(stats_part.p, pb, stats.p);
  TABI_CUDA(cudaMemcpyAsync(h_stats, stats.p, sizeof(double) * 8, cudaMemcpyDeviceToHost, s));
  TABI_CUDA(cudaStreamSynchronize(s));
  const double abar = h_stats[0] / n;
  TABI_REQUIRE(abar > 0.0 && std::isfinite(h_stats[1]), TABI_ERR_ARG,
               "warm start: panel areas must be positive and b finite");
  // cells of ~2K panels' worth of area: the K nearest lie within a few cells
  Grid g;
  g.x0 = (float)h_stats[2];
  g.y0 = (float)h_stats[3];
  g.z0 = (float)h_stats[4];
  const double ext[3] = {h_stats[5] - h_stats[2], h_stats[6] - h_stats[3],
                         h_stats[7] - h_stats[4]};
  double h = std::sqrt(2.0 * kK * abar / kPi);
  auto dims = [&](double hh, int d) { return std::max(1, (int)std::ceil(ext[d] / hh + 1e-6)); };
  while ((double)dims(h, 0) * dims(h, 1) * dims(h, 2) > 8.0e6) h *= 1.25;
  g.h = (float)h;
  g.nx = dims(h, 0);
  g.ny = dims(h, 1);
  g.nz = dims(h, 2);
  const int nc = g.nx * g.ny * g.nz;
  cell.alloc(n);
  ccnt.alloc(nc + 1);
  coff.alloc(nc + 1);
  csorted.alloc(n);
  const int sb = ceil_div(nc, kScanB);
  const int rb = ceil_div(n, kScanB);
  sbuf.alloc(std::max(sb, rb) + 2);
  TABI_CUDA(cudaMemsetAsync(ccnt.p, 0, sizeof(int) * (nc + 1), s));
  ws_cell_count_kernel<<<ceil_div(n, 256), 256, 0, s>>>(n, pos.p, g, cell.p, ccnt.p);
  ws_scan_block_kernel<<<sb, kScanB, 0, s>>>(ccnt.p, nc, coff.p, sbuf.p);
  ws_scan_sums_kernel<<<1, 32, 0, s>>>(sbuf.p, sb, sbuf.p + sb);
  ws_scan_add_kernel<<<sb, kScanB, 0, s>>>(coff.p, nc, sbuf.p, sbuf.p + sb);
  TABI_CUDA(cudaMemcpyAsync(ccnt.p, coff.p, sizeof(int) * nc, cudaMemcpyDeviceToDevice, s));
  ws_cell_fill_kernel<<<ceil_div(n, 256), 256, 0, s>>>(n, cell.p, ccnt.p, csorted.p);
  nbr.alloc((size_t)n * kK);
  err.alloc(1);
  TABI_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));
  ws_knn_kernel<<<ceil_div(n, 128), 128, 0, s>>>(n, pos.p, g, coff.p, csorted.p, nbr.p, err.p);
  // reversed lists
  rcnt.alloc(n + 1);
  roff.alloc(n + 1);
  rev.alloc((size_t)n * kK);
  TABI_CUDA(cudaMemsetAsync(rcnt.p, 0, sizeof(int) * (n + 1), s));
  ws_rev_count_kernel<<<ceil_div((int64_t)n * kK, 256), 256, 0, s>>>(n, nbr.p, rcnt.p);
  ws_scan_block_kernel<<<rb, kScanB, 0, s>>>(rcnt.p, n, roff.p, sbuf.p);
  ws_scan_sums_kernel<<<1, 32, 0, s>>>(sbuf.p, rb, sbuf.p + rb);
  ws_scan_add_kernel<<<rb, kScanB, 0, s>>>(roff.p, n, sbuf.p, sbuf.p + rb);
  TABI_CUDA(cudaMemcpyAsync(rcnt.p, roff.p, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
  ws_rev_fill_kernel<<<ceil_div((int64_t)n * kK, 256), 256, 0, s>>>(n, nbr.p, rcnt.p, rev.p);
  ws_rev_sort_kernel<<<ceil_div(n, 128), 128, 0, s>>>(n, roff.p, rev.p);
  // node features
  dbar.alloc(n);
  feat.alloc((size_t)n * kF);
  ws_node_kernel<<<ceil_div(n, 128), 128, 0, s>>>(n, pos.p, nrm.p, bfl.p, zfl.p, nbr.p, stats.p,
                                                  dbar.p, feat.p);
  TABI_CUDA(cudaGetLastError());
}

void WsNet::dw(int M, int Kd, int N, const float* A, const float* D, float* g, cudaStream_t s) {
  // rows per chunk: two blocks for each SM, between 64 and 1,024
  const int chunk = std::min(1024, std::max(64, ceil_div(ceil_div(M, 2 * kSMs), kGK) * kGK));
  const int nch = ceil_div(M, chunk);
  part.alloc((size_t)nch * Kd * N);
  auto launch = [&](auto t) {
    constexpr int T = decltype(t)::value;
    dim3 grid(ceil_div(Kd, 16 * T), ceil_div(N, 16 * T), nch);
    ws_dw_kernel<T><<<grid, 256, 0, s>>>(M, Kd, N, chunk, A, Kd, D, N, part.p);
  };
  if (Kd == N)
    with_tile(N, launch);
  else
    launch(std::integral_constant<int, 2>());  // the input and output layers
  sum_parts(part.p, nch, (int64_t)Kd * N, g, s);
}

void WsNet::colsum(int M, int N, const float* X, float* g, cudaStream_t s) {
  part2.alloc((size_t)kRedB * N);
  ws_colsum_kernel<<<kRedB, 256, 0, s>>>(M, N, X, part2.p);
  sum_parts(part2.p, kRedB, N, g, s);
}

void WsNet::forward(const WsInput& in, double* xout, const double* target, cudaStream_t s) {
  const int n = in.n;
  graph(in, s);
  const size_t nh = (size_t)n * H;
  hs.alloc(nh * (L + 1));
  us.alloc(nh * L);
  as.alloc(nh * L);
  zs.alloc(nh * L);
  pre0.alloc(nh);
  const __nv_bfloat16* W = wbf.p;
  const float* T = theta.p;
  gemm<false, 3>(n, H, kF, feat.p, kF, W + off_W0, H, T + off_b0, hs.p, H, pre0.p, nullptr, s);
  for (int l = 0; l < L; ++l) {
    const Layer& y = lay[l];
    float* h = hs.p + nh * l;
    float* u = us.p + nh * l;
    float* a = as.p + nh * l;
    float* z = zs.p + nh * l;
    gemm<false, 0>(n, H, H, h, H, W + y.Wa, H, nullptr, u, H, nullptr, nullptr, s);
    ws_agg_fwd_kernel<<<ceil_div(n, kWsNodes), H, 0, s>>>(n, H, pos.p, nrm.p, dbar.p, nbr.p,
                                                           W + y.Wf, T + y.bf, u, a);
    gemm<false, 1>(n, H, H, h, H, W + y.Wb1, H, T + y.bb, z, H, nullptr, nullptr, s);
    gemm<false, 4>(n, H, H, a, H, W + y.Wb2, H, nullptr, h + nh, H, z, h, s);
  }
  dout.alloc(2 * (size_t)n);
  lpart.alloc(kRedB + 2);
  ws_head_kernel<<<kRedB, 256, 0, s>>>(n, H, hs.p + nh * L, W + off_Wo, T + off_bo, in.b, in.z,
                                       stats.p, xout, target, dout.p, lpart.p);
  if (target) ws_loss_final_kernel<<<1, 32, 0, s>>>(lpart.p, kRedB, n, lpart.p + kRedB);
  TABI_CUDA(cudaGetLastError());
}

void WsNet::backward(int n, cudaStream_t s) {
  const size_t nh = (size_t)n * H;
  dh.alloc(nh);
  dz.alloc(nh);
  da.alloc(nh);
  du.alloc(nh);
  wpart.alloc((size_t)kWsBlocks * (kE + 1) * H);
  float* G = grad.p;
  const __nv_bfloat16* W = wbf.p;
  const float* T = theta.p;
  TABI_CUDA(cudaMemsetAsync(G, 0, sizeof(float) * np, s));
  // head
  dw(n, H, 2, hs.p + nh * L, dout.p, G + off_Wo, s);
  colsum(n, 2, dout.p, G + off_bo, s);
  ws_head_bwd_kernel<<<1024, 256, 0, s>>>(n, H, dout.p, W + off_Wo, dh.p);
  const int eb = 1024;
  for (int l = L - 1; l >= 0; --l) {
    const Layer& y = lay[l];
    const float* hin = hs.p + nh * l;
    const float* u = us.p + nh * l;
    const float* a = as.p + nh * l;
    const float* z = zs.p + nh * l;
    ws_dsilu_kernel<<<eb, 256, 0, s>>>((int64_t)nh, dh.p, z, dz.p);
    dw(n, H, H, hin, dz.p, G + y.Wb1, s);
    dw(n, H, H, a, dz.p, G + y.Wb2, s);
    colsum(n, H, dz.p, G + y.bb, s);
    // dh_in = dh + dz Wb1^T ; da = dz Wb2^T
    gemm<true, 2>(n, H, H, dz.p, H, W + y.Wb1, H, nullptr, dh.p, H, nullptr, nullptr, s);
    gemm<true, 0>(n, H, H, dz.p, H, W + y.Wb2, H, nullptr, da.p, H, nullptr, nullptr, s);
    // aggregation: Wf (kE x H) and bf (H) are adjacent in the flat layout
    ws_agg_bwd_w_kernel<<<kWsBlocks, H, 0, s>>>(n, H, pos.p, nrm.p, dbar.p, nbr.p, W + y.Wf,
                                                T + y.bf, u, da.p, wpart.p);
    sum_parts(wpart.p, kWsBlocks, (int64_t)(kE + 1) * H, G + y.Wf, s);
    ws_agg_bwd_u_kernel<<<ceil_div(n, kWsNodes), H, 0, s>>>(n, H, pos.p, nrm.p, dbar.p, roff.p,
                                                             rev.p, W + y.Wf, T + y.bf, da.p,
                                                             du.p);
    dw(n, H, H, hin, du.p, G + y.Wa, s);
    gemm<true, 2>(n, H, H, du.p, H, W + y.Wa, H, nullptr, dh.p, H, nullptr, nullptr, s);
  }
  // input layer
  ws_dsilu_kernel<<<eb, 256, 0, s>>>((int64_t)nh, dh.p, pre0.p, dz.p);
  dw(n, kF, H, feat.p, dz.p, G + off_W0, s);
  colsum(n, H, dz.p, G + off_b0, s);
  TABI_CUDA(cudaGetLastError());
}

void WsNet::adam(double lr, cudaStream_t s) {
  ++adam_t;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)adam_t), c2 = 1.f - std::pow(b2, (float)adam_t);
  ws_adam_kernel<<<256, 256, 0, s>>>(np, theta.p, grad.p, m.p, v.p, (float)lr, b1, b2, c1, c2,
                                     1e-8f, wbf.p);
  TABI_CUDA(cudaGetLastError());
}

double WsNet::read_loss(cudaStream_t s) {
  TABI_CUDA(cudaMemcpyAsync(h_stats + 8, lpart.p + kRedB, sizeof(double), cudaMemcpyDeviceToHost,
                            s));
  TABI_CUDA(cudaStreamSynchronize(s));
  return h_stats[8];
}

bool WsNet::graph_exact(cudaStream_t s) {
  int e = 0;
  TABI_CUDA(cudaMemcpyAsync(&h_stats[9], err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  TABI_CUDA(cudaStreamSynchronize(s));
  std::memcpy(&e, &h_stats[9], sizeof(int));
  return e == 0;
}

}  // namespace tabi
