// matvec.cu -- the treecode operator y = A x (TREE_COMPP_PB,
// treecode3d_pb.f:1130-1189) as four device steps:
//
//  1. moments   COMP_MS (treecode3d_pb.f:859-916) for every cluster some
//               target accepts.  FP64: the coefficients of its two harmonic
//               polynomials per degree (harmonic.cuh).  FP32: the 16 source
//               charges of pb_kernel (main.f90:664-694) reduce to 4 distinct
//               ones -- A*x2 and (n_d*A)*x1 -- so 4 raw moment sets are
//               summed, then weighted by the integer part of der_cof
//               (main.f90:380-399) into the 16 per-index sets the contraction
//               reads.
//  2. far       one thread per (target, accepted cluster), cluster moments
//               staged in shared memory: COMP_TCOEFF + COMPP_TREE_PB in solid
//               harmonics (FP64, harmonic.cuh) or as the generated Cartesian
//               recurrence (FP32, taylor_gen.cuh).
//  3. near      one thread per (target, near leaf): COMPP_DIRECT_PB
//               (treecode3d_pb.f:919-1008) over the leaf's faces staged in
//               shared memory; the target's own face is skipped, which is what
//               the reference's shift-and-zero-area trick (:1169-1172) amounts
//               to.
//  4. reduce    per target, the interaction results summed in traversal order:
//               y1 = pre1*x1 - peng1, y2 = pre2*x2 - peng2 (:1177-1178).
// All results are written to per-(target, interaction) slots fixed by the
// traversal, so the sums are deterministic.
#include <algorithm>
#include <type_traits>

#include "bie_kernels.cuh"
#include "fast_math.cuh"
#include "harmonic.cuh"
#include "reduce.cuh"
#include "taylor_gen.cuh"
#include "tabi_impl.cuh"

namespace tabi {

namespace {

// ---- moments
// Cartesian moments of the mixed-precision far field, summed in FP64.  A group
// of G threads takes a chunk of up to 256 sources of a cluster, a thread S of the 4
// raw sets of a term: the powers of 64 sources at a time and the 4 charges lie in
// shared memory, and with S = 4 seven shared words serve 4 sums, with S = 1 four
// words each sum.  Every sum runs over its chunk's sources in order, so S changes
// no bit.  S = 1 up to order 5 while there are few (source, term) pairs (kMomFew),
// where the length of a thread's loop counts and not its loads: order 3, leaves of
// up to 400, S = 1 and 4: 1,098 faces 5.9 and 9.5 us, 11,184 faces 8.8 and 17.0,
// 28,550 faces 22.0 and 19.8; order 5, 7,328 faces 10.4 and 11.8, 11,184 faces 13.6
// and 12.1; order 6, 7,328 faces 17.7 and 14.3.
template <int P, int S>
struct MomShape {
  static constexpr int NT = tabi_nterms(P), W = 3 * (P + 1) + 4, TILE = S == 1 ? 128 : 64;
  static constexpr int G = (NT * (4 / S) + 31) / 32 * 32;
  static constexpr int CPB = S == 1 || G >= 128 ? 1 : 128 / G;
  static constexpr int PITCH = S == 1 ? W : (W + 1) / 2 * 2;  // S = 4: 16-byte aligned rows
};
constexpr int64_t kMomFew = 400000;

template <int P, int S>
__global__ void __launch_bounds__(MomShape<P, S>::G* MomShape<P, S>::CPB) mom_partial_kernel(
    const int4* __restrict__ chunks, int nchunk, const int* __restrict__ mslot_node,
    const double* __restrict__ nd_mid, const double* __restrict__ px,
    const double* __restrict__ py, const double* __restrict__ pz, const double* __restrict__ nx,
    const double* __restrict__ ny, const double* __restrict__ nz,
    const double* __restrict__ area, const double* __restrict__ x, int n,
    double* __restrict__ mraw) {
  using M = MomShape<P, S>;
  constexpr int NT = M::NT, TILE = M::TILE, G = M::G;
  __shared__ __align__(16) double stage[M::CPB][TILE][M::PITCH];
  const int g = threadIdx.x / G, t = threadIdx.x % G;
  const int set0 = t / NT, term = t - set0 * NT;  // S = 4: set0 is 0 for every term
  const bool own = t < NT * (4 / S);
  const int c = blockIdx.x * M::CPB + g;
  const int4 ch = c < nchunk ? chunks[c] : make_int4(0, 0, 0, 0);
  const int node = mslot_node[ch.x];
  const double mx = nd_mid[3 * node], my = nd_mid[3 * node + 1], mz = nd_mid[3 * node + 2];
  double(*st)[M::PITCH] = stage[g];
  int k1 = 0, k2 = 0, k3 = 0;
  if (own) {
    const signed char(*tt)[3] = tabi_terms<P>();
    k1 = 4 + tt[term][0];
    k2 = 4 + P + 1 + tt[term][1];
    k3 = 4 + 2 * (P + 1) + tt[term][2];
  }
  double acc[S] = {};
  for (int base = 0; base < 256; base += TILE) {
    const int cnt = min(TILE, ch.z - base);
    if (__syncthreads_and(cnt <= 0)) break;
    for (int q = t; q < cnt; q += G) {
      const int i = ch.y + base + q;
      // COMP_MS :876-889: dx = x - mid, powers by repeated multiplication
      const double dx = px[i] - mx, dy = py[i] - my, dz = pz[i] - mz;
      double a = 1.0, b = 1.0, d = 1.0;
#pragma unroll
      for (int p = 0; p <= P; ++p) {
        st[q][4 + p] = a;
        st[q][4 + P + 1 + p] = b;
        st[q][4 + 2 * (P + 1) + p] = d;
        a *= dx;
        b *= dy;
        d *= dz;
      }
      const double A = area[i], x1 = x[i], x2 = x[n + i];
      // pb_kernel (main.f90:673-681): A*x2 and (n_d*A)*x1
      st[q][0] = A * x2;
      st[q][1] = (nx[i] * A) * x1;
      st[q][2] = (ny[i] * A) * x1;
      st[q][3] = (nz[i] * A) * x1;
    }
    __syncthreads();
    if (own)
#pragma unroll 4
      for (int q = 0; q < cnt; ++q) {
        const double txyz = st[q][k1] * st[q][k2] * st[q][k3];
        if constexpr (S == 1) {
          acc[0] = fma(st[q][set0], txyz, acc[0]);
        } else {
          const double2 s0 = *reinterpret_cast<const double2*>(&st[q][0]);
          const double2 s1 = *reinterpret_cast<const double2*>(&st[q][2]);
          acc[0] = fma(s0.x, txyz, acc[0]);
          acc[1] = fma(s0.y, txyz, acc[1]);
          acc[2] = fma(s1.x, txyz, acc[2]);
          acc[3] = fma(s1.y, txyz, acc[3]);
        }
      }
  }
  if (c < nchunk && own)
#pragma unroll
    for (int k = 0; k < S; ++k) mraw[((size_t)ch.w * 4 + set0 + k) * NT + term] = acc[k];
}

// the 16 weighted sets (kk and der_cof, main.f90:358-399) in the order the far
// field reads them, from the chunks' sums in order
template <int P>
__global__ void __launch_bounds__(256) mom_final_kernel(const int2* __restrict__ mslot_chunks,
                                                        const double* __restrict__ mraw,
                                                        float* __restrict__ mw) {
  constexpr int NT = tabi_nterms(P);
  __shared__ double raw[4 * NT];
  const int2 cr = mslot_chunks[blockIdx.x];
  for (int q = threadIdx.x; q < 4 * NT; q += blockDim.x) {
    double v = 0.0;
    for (int c = 0; c < cr.y; ++c) v += mraw[(size_t)(cr.x + c) * 4 * NT + q];
    raw[q] = v;
  }
  __syncthreads();
  const unsigned short* mpos = tabi_mpos<P>();
  const signed char* mwgt = tabi_mwgt<P>();
  for (int q = threadIdx.x; q < 16 * NT; q += blockDim.x) {
    const int idx = q / NT, term = q - idx * NT;
    const int set = idx == 0 ? 0 : idx <= 3 ? idx : idx <= 6 ? 0 : 1 + (idx - 7) / 3;
    mw[(size_t)blockIdx.x * 16 * NT + mpos[q]] = (float)((double)mwgt[q] * raw[set * NT + term]);
  }
}

// FP64 moments.  One block per chunk of up to 256 sources of a cluster; a warp
// takes 32 sources at a time, each thread evaluates one source's
// contributions to the 2 (p+2)^2 sums into its row of the warp's tile, and the
// lanes add up the tile's columns.  One evaluation serves all sums: the form
// with a thread per sum and three staged power factors per source ran
// 4 C(p+3,3) threads of 7 shared loads a source.
constexpr int harm_warps(int p) { return p <= 4 ? 4 : 2; }
constexpr size_t harm_mom_smem(int p) {
  return sizeof(double) * harm_warps(p) * 32 * (harm_raw(p) + 1);
}

template <int P>
__global__ void __launch_bounds__(32 * harm_warps(P)) harm_mom_kernel(
    const int4* __restrict__ chunks, const int* __restrict__ mslot_node,
    const double* __restrict__ nd_mid, const double* __restrict__ px,
    const double* __restrict__ py, const double* __restrict__ pz, const double* __restrict__ nx,
    const double* __restrict__ ny, const double* __restrict__ nz,
    const double* __restrict__ area, const double* __restrict__ x, int n,
    const HarmBeta<P> beta, double eps, double* __restrict__ mraw) {
  constexpr int NC = harm_raw(P), PITCH = NC + 1, W = harm_warps(P);
  constexpr int CPL = (NC + 31) / 32;  // columns per lane
  extern __shared__ double hsm[];
  const int4 ch = chunks[blockIdx.x];
  const int node = mslot_node[ch.x];
  const double mx = nd_mid[3 * node], my = nd_mid[3 * node + 1], mz = nd_mid[3 * node + 2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* tile = hsm + warp * 32 * PITCH;
  double acc[CPL];
#pragma unroll
  for (int k = 0; k < CPL; ++k) acc[k] = 0.0;
  for (int base = 32 * warp; base < ch.z; base += 32 * W) {
    const int cnt = min(32, ch.z - base);
    if (lane < cnt) {
      const int i = ch.y + base + lane;
      const double A = area[i], x1 = x[i], x2 = x[n + i];
      // pb_kernel (main.f90:673-681): A*x2 and (n_d*A)*x1
      harm_source<P>(px[i] - mx, py[i] - my, pz[i] - mz, A * x2, (nx[i] * A) * x1,
                     (ny[i] * A) * x1, (nz[i] * A) * x1, beta, eps,
                     tile + lane * PITCH);
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
      const int c = lane + 32 * k;
      if (c < NC)
        for (int q = 0; q < cnt; ++q) acc[k] += tile[q * PITCH + c];
    }
    __syncwarp();
  }
#pragma unroll
  for (int k = 0; k < CPL; ++k)
    if (lane + 32 * k < NC) tile[lane + 32 * k] = acc[k];
  __syncthreads();
  for (int c = threadIdx.x; c < NC; c += 32 * W) {
    double v = hsm[c];
#pragma unroll
    for (int w = 1; w < W; ++w) v += hsm[w * 32 * PITCH + c];
    mraw[(size_t)ch.w * NC + c] = v;
  }
}

// one block per cluster: the chunks' sums in order, the constants of (l, m),
// and the gradients' coefficients, in the order harm_eval reads them
template <int P>
__global__ void __launch_bounds__(128) harm_final_kernel(const int2* __restrict__ mslot_chunks,
                                                         const double* __restrict__ mraw,
                                                         double* __restrict__ mw) {
  constexpr int NC = harm_raw(P), NE = (P + 2) * (P + 2);
  __shared__ double c[NC], sa[(P + 2) * (P + 3) / 2];
  const int2 cr = mslot_chunks[blockIdx.x];
  auto degree = [](int e) {
    int l = 0;
    while ((l + 1) * (l + 1) <= e) ++l;
    return l;
  };
  for (int q = threadIdx.x; q < (P + 2) * (P + 3) / 2; q += blockDim.x) {
    int l = 0;
    while ((l + 1) * (l + 2) / 2 <= q) ++l;
    sa[q] = harm_a(l, q - l * (l + 1) / 2);
  }
  for (int q = threadIdx.x; q < NC; q += blockDim.x) {
    double raw = 0.0;
    for (int k = 0; k < cr.y; ++k) raw += mraw[(size_t)(cr.x + k) * NC + q];
    const int e = q >> 1, l = degree(e), m = (e - l * l + 1) >> 1;
    c[q] = raw * harm_scale(l, m, q & 1);
  }
  __syncthreads();
  double* out = mw + (size_t)blockIdx.x * harm_size(P);
  for (int q = threadIdx.x; q < 8 * NE; q += blockDim.x) {
    const int e = q >> 3, f = q & 7, l = degree(e), r = e - l * l, m = (r + 1) >> 1;
    const double a = sa[l * (l + 1) / 2 + m];
    if (l <= P)
      out[q] = a * (f < 2 ? c[2 * e + f]
                          : harm_grad(c + (f < 5 ? 0 : 1), l, m, r > 0 && !(r & 1), (f - 2) % 3));
    else if (f < 2)
      out[8 * (P + 1) * (P + 1) + 2 * r + f] = a * c[2 * e + f];
  }
}

// ---- far field
// FP64 (harmonic.cuh): one block per (cluster, up to 64 NT of its targets), NT =
// far_nt targets per thread, which share every coefficient's shared load.

template <int P, int NT>
__global__ void __launch_bounds__(kFarThreads) far_harm_kernel(
    const WorkItem* __restrict__ work, const int2* __restrict__ ent,
    const double* __restrict__ mw, const double* __restrict__ nd_mid,
    const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
    const double* __restrict__ nx, const double* __restrict__ ny, const double* __restrict__ nz,
    double kappa, double inv_eps, double2* __restrict__ res) {
  __shared__ __align__(16) double sm[harm_size(P)];
  const WorkItem wi = work[blockIdx.x];
  const double* src = mw + (size_t)wi.mslot * harm_size(P);
  for (int q = threadIdx.x; q < harm_size(P) / 2; q += kFarThreads)
    reinterpret_cast<double2*>(sm)[q] = reinterpret_cast<const double2*>(src)[q];
  const double mx = nd_mid[3 * wi.node], my = nd_mid[3 * wi.node + 1], mz = nd_mid[3 * wi.node + 2];
  double x[NT], y[NT], z[NT], n0[NT], n1[NT], n2[NT], o1[NT], o2[NT];
  int slot[NT];
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    // a thread past the end repeats the last target and writes nothing
    const int2 e = ent[wi.start + min((int)threadIdx.x + kFarThreads * k, wi.count - 1)];
    slot[k] = e.y;
    // COMP_TCOEFF :707-709: target - mid
    x[k] = px[e.x] - mx;
    y[k] = py[e.x] - my;
    z[k] = pz[e.x] - mz;
    n0[k] = nx[e.x];
    n1[k] = ny[e.x];
    n2[k] = nz[e.x];
  }
  __syncthreads();
  if ((int)(threadIdx.x & ~31u) >= wi.count) return;  // a warp without targets
  harm_eval<P, NT>(x, y, z, n0, n1, n2, kappa, inv_eps, sm, o1, o2);
#pragma unroll
  for (int k = 0; k < NT; ++k)
    if ((int)threadIdx.x + kFarThreads * k < wi.count)
      res[slot[k]] = make_double2(o1[k] * kOneOver4Pi, o2[k] * kOneOver4Pi);
}

// FP32 (mixed precision): the target-to-centre offset is formed in FP64 and
// rounded once, the Taylor recurrences and the contraction run in FP32, the
// result is widened to FP64 for the per-target sum.  Bound by the latency of
// its straight-line code at a few warps per SM, so the register cap is where
// more warps stop paying for the spills: far field at orders 3, 4, 5, 6 and 8
// 232 -> 212, 575 -> 389, 967 -> 723, 1,239 -> 1,131 and 2,092 -> 1,493 us;
// order 7 is fastest without one (863, 919 at 168 registers).
constexpr int far_blocks(int p) {
  return p == 3 ? 12 : p == 4 || p == 5 ? 8 : p == 6 || p == 8 ? 6 : 1;
}

template <int P>
__global__ void __launch_bounds__(kFarThreads, far_blocks(P)) far_kernel(const WorkItem* __restrict__ work,
                                                 const int2* __restrict__ ent,
                                                 const float* __restrict__ mw,
                                                 const double* __restrict__ nd_mid,
                                                 const double* __restrict__ px,
                                                 const double* __restrict__ py,
                                                 const double* __restrict__ pz,
                                                 const double* __restrict__ nx,
                                                 const double* __restrict__ ny,
                                                 const double* __restrict__ nz, float kappa,
                                                 float eps, double2* __restrict__ res) {
  constexpr int NT = tabi_nterms(P);
  __shared__ float4 smw[4 * NT];
  WorkItem wi = work[blockIdx.x];
  const float4* src = reinterpret_cast<const float4*>(mw + (size_t)wi.mslot * 16 * NT);
  for (int q = threadIdx.x; q < 4 * NT; q += blockDim.x) smw[q] = src[q];
  __syncthreads();
  for (int k = threadIdx.x; k < wi.count; k += blockDim.x) {
    const int2 e = ent[wi.start + k];
    const int t = e.x;
    // COMP_TCOEFF :707-709: dx = target - mid
    const float dx = (float)(px[t] - nd_mid[3 * wi.node]);
    const float dy = (float)(py[t] - nd_mid[3 * wi.node + 1]);
    const float dz = (float)(pz[t] - nd_mid[3 * wi.node + 2]);
    float o1, o2;
    far_eval<P, float>(dx, dy, dz, kappa, smw, (float)nx[t], (float)ny[t], (float)nz[t], eps,
                       1.f / eps, o1, o2);
    res[e.y] = make_double2((double)o1 * kOneOver4Pi, (double)o2 * kOneOver4Pi);
  }
}

// ---- near field
// FP64: one block per (leaf, up to 128/S of the targets that meet it), S
// neighbouring threads per target, each over every S-th of the leaf's faces.
// Bound by the FP64 pipe, so the four kernels are formed as sums over the
// weighted sources (m = A x1 n, w = A x2, d = r - s, i = 1/|d|,
// t = (1 + kappa r) e, e = e^{-kappa r}):
//   y1: i (i^2 (m.d)(1 - eps t) + w (1 - e)),
//   y2: i^3 ((m.v0 - 3 i^2 (m.d)(v0.d))(t - 1) - kappa^2 (m.d)(v0.d) e
//            + w (v0.d)(1 - t/eps)),
// times 1/(4 pi) at the end: 37 FP64 instructions beside the reciprocal root and
// the exponential (fast_math.cuh), against 45 of the factored form of each
// kernel.  Only blocks in which a target meets its own leaf, or kappa times a
// distance may leave the exponential's table, test for either in the loop.
// Measured beside the far field, 73.5 M pairs: 0.50 -> 0.32 ms; 193 M
// pairs: 1.36 -> 0.90 ms; 0.55 M pairs (1,272 targets, one thread each gave 27
// blocks): 49 -> 20 us.
constexpr int kNearThreads = 128;
constexpr int kNearTile = 256;

template <int S, bool CHECK>
__device__ __forceinline__ void near_tile(const double2 (*src)[4], const double* tab, int cnt,
                                          int self, double tx, double ty, double tz, double vx,
                                          double vy, double vz, double kappa, double eps,
                                          double inv_eps, double& p1, double& p2) {
  const double k2 = kappa * kappa;
#pragma unroll 4
  for (int q = (int)threadIdx.x % S; q < cnt; q += S) {
    const double2 a = src[q][0], b = src[q][1], c = src[q][2], g = src[q][3];
    double dx = a.x - tx, dy = a.y - ty, dz = b.x - tz;
    double mx = c.x, my = c.y, mz = g.x, w = b.y;
    if (CHECK && q == self) {  // the own face: no contribution, and no 1/0
      dx = 1.0;
      mx = my = mz = w = 0.0;
    }
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const double i = fast_rsqrt(r2), i2 = i * i;
    const double kr = kappa * (r2 * i);
    const double e = exp_neg<CHECK>(kr, tab);
    const double t = fma(kr, e, e);
    const double md = fma(mx, dx, fma(my, dy, mz * dz));
    const double vd = fma(vx, dx, fma(vy, dy, vz * dz));
    const double mv = fma(mx, vx, fma(my, vy, mz * vz));
    p1 = fma(i, fma(i2 * md, fma(-eps, t, 1.0), fma(-e, w, w)), p1);
    const double mvd = md * vd;
    double s = fma(-3.0 * i2, mvd, mv) * (t - 1.0);
    s = fma(-(k2 * e), mvd, s);
    s = fma(w * vd, fma(-inv_eps, t, 1.0), s);
    p2 = fma(i * i2, s, p2);
  }
}

template <int S>
__global__ void __launch_bounds__(kNearThreads, 5) near_kernel(
    const WorkItem* __restrict__ work, const int2* __restrict__ ent,
    const int* __restrict__ nd_ibeg, const int* __restrict__ nd_num,
    const double* __restrict__ nd_mid, const double* __restrict__ nd_rad,
    const double* __restrict__ px, const double* __restrict__ py,
    const double* __restrict__ pz, const double* __restrict__ nx,
    const double* __restrict__ ny, const double* __restrict__ nz,
    const double* __restrict__ area, const double* __restrict__ x, int n, double kappa,
    double eps, double2* __restrict__ res) {
  // per face: (x, y), (z, A x2), (A x1 n_x, A x1 n_y), (A x1 n_z, -)
  __shared__ double2 src[kNearTile][4];
  __shared__ double tab[kExpTab];
  exp_table_fill(tab);
  const WorkItem wi = work[blockIdx.x];
  const int ib = nd_ibeg[wi.node], nsrc = nd_num[wi.node];
  const int k = (int)threadIdx.x / S;
  const bool own = k < wi.count;
  const int2 ent_k = ent[wi.start + min(k, wi.count - 1)];
  const int t = ent_k.x;
  const double tx = px[t], ty = py[t], tz = pz[t], vx = nx[t], vy = ny[t], vz = nz[t];
  const double far_end =
      sqrt((tx - nd_mid[3 * wi.node]) * (tx - nd_mid[3 * wi.node]) +
           (ty - nd_mid[3 * wi.node + 1]) * (ty - nd_mid[3 * wi.node + 1]) +
           (tz - nd_mid[3 * wi.node + 2]) * (tz - nd_mid[3 * wi.node + 2])) +
      nd_rad[wi.node];  // no face of the leaf is further from the target
  const bool check = __syncthreads_or((t >= ib && t < ib + nsrc) ||
                                      !(kappa * far_end < 0.99 * kExpTabEnd));
  const double inv_eps = 1.0 / eps;
  double p1 = 0.0, p2 = 0.0;
  for (int b0 = 0; b0 < nsrc; b0 += kNearTile) {
    const int cnt = min(kNearTile, nsrc - b0);
    if (b0 > 0) __syncthreads();
    for (int q = threadIdx.x; q < cnt; q += kNearThreads) {
      const int j = ib + b0 + q;
      const double A = area[j], w1 = A * x[j];
      src[q][0] = make_double2(px[j], py[j]);
      src[q][1] = make_double2(pz[j], A * x[n + j]);
      src[q][2] = make_double2(w1 * nx[j], w1 * ny[j]);
      src[q][3] = make_double2(w1 * nz[j], 0.0);
    }
    __syncthreads();
    if (own) {
      if (check)
        near_tile<S, true>(src, tab, cnt, t - (ib + b0), tx, ty, tz, vx, vy, vz, kappa, eps,
                           inv_eps, p1, p2);
      else
        near_tile<S, false>(src, tab, cnt, 0, tx, ty, tz, vx, vy, vz, kappa, eps, inv_eps, p1,
                            p2);
    }
  }
#pragma unroll
  for (int o = S / 2; o > 0; o >>= 1) {
    p1 += __shfl_xor_sync(0xffffffffu, p1, o);
    p2 += __shfl_xor_sync(0xffffffffu, p2, o);
  }
  if (own && threadIdx.x % S == 0)
    res[ent_k.y] = make_double2(p1 * kOneOver4Pi, p2 * kOneOver4Pi);
}

// Mixed-precision near field.  Each face's position relative to the centre of
// its leaf is kept as an unevaluated FP32 sum hi + lo (to ~2^-48 of the leaf
// size), with its area and its normal in FP32 (leaf_rel_kernel, once per tree);
// the target is split the same way against the same centre.  r - s is then
// (hi_s - hi_t) + (lo_s - lo_t), accurate to FP32 rounding of |r - s| itself:
// with one rounded FP32 coordinate, n.(r - s) of adjacent panels (a few
// hundredths of an Angstrom on a curved surface) would carry the 1e-6 A
// rounding of leaf-sized coordinates, an error of ~1e-4 relative in K1 and K4.
// The four kernels and the per-(target, leaf) sum run in FP32; the per-target
// sum over leaves stays FP64 (reduce_kernel).
__global__ void leaf_rel_kernel(const int* __restrict__ leaves, const int* __restrict__ nd_ibeg,
                                const int* __restrict__ nd_num, const double* __restrict__ nd_mid,
                                const double* __restrict__ px, const double* __restrict__ py,
                                const double* __restrict__ pz, const double* __restrict__ nx,
                                const double* __restrict__ ny, const double* __restrict__ nz,
                                const double* __restrict__ area, float4* __restrict__ lpos,
                                float4* __restrict__ llo, float4* __restrict__ lnrm) {
  const int node = leaves[blockIdx.x];
  const int ib = nd_ibeg[node], m = nd_num[node];
  const double mx = nd_mid[3 * node], my = nd_mid[3 * node + 1], mz = nd_mid[3 * node + 2];
  for (int q = threadIdx.x; q < m; q += blockDim.x) {
    const int j = ib + q;
    const double rx = px[j] - mx, ry = py[j] - my, rz = pz[j] - mz;
    const float hx = (float)rx, hy = (float)ry, hz = (float)rz;
    lpos[j] = make_float4(hx, hy, hz, (float)area[j]);
    llo[j] = make_float4((float)(rx - hx), (float)(ry - hy), (float)(rz - hz), 0.f);
    lnrm[j] = make_float4((float)nx[j], (float)ny[j], (float)nz[j], 0.f);
  }
}

constexpr int kNearTileF = 512;

__global__ void __launch_bounds__(kNearThreads) near_kernel_f32(
    const WorkItem* __restrict__ work, const int2* __restrict__ ent,
    const int* __restrict__ nd_ibeg, const int* __restrict__ nd_num,
    const double* __restrict__ nd_mid, const double* __restrict__ px,
    const double* __restrict__ py, const double* __restrict__ pz,
    const float4* __restrict__ lpos, const float4* __restrict__ llo,
    const float4* __restrict__ lnrm, const double* __restrict__ x, int n, float kappa,
    float eps, double2* __restrict__ res) {
  __shared__ float4 s_p[kNearTileF];  // relative position (hi), A * x1
  __shared__ float4 s_l[kNearTileF];  // relative position (lo)
  __shared__ float4 s_n[kNearTileF];  // normal, A * x2
  WorkItem wi = work[blockIdx.x];
  const int ib = nd_ibeg[wi.node], nsrc = nd_num[wi.node];
  const bool own = (int)threadIdx.x < wi.count;
  int t = 0, slot = 0;
  float tx = 0.f, ty = 0.f, tz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  float vx = 0.f, vy = 0.f, vz = 0.f;
  if (own) {
    int2 e = ent[wi.start + threadIdx.x];
    t = e.x;
    slot = e.y;
    const double rx = px[t] - nd_mid[3 * wi.node];
    const double ry = py[t] - nd_mid[3 * wi.node + 1];
    const double rz = pz[t] - nd_mid[3 * wi.node + 2];
    tx = (float)rx;
    ty = (float)ry;
    tz = (float)rz;
    lx = (float)(rx - tx);
    ly = (float)(ry - ty);
    lz = (float)(rz - tz);
    float4 nv = lnrm[t];
    vx = nv.x;
    vy = nv.y;
    vz = nv.z;
  }
  const float inv_eps = 1.f / eps;
  float p1 = 0.f, p2 = 0.f;
  for (int b0 = 0; b0 < nsrc; b0 += kNearTileF) {
    const int cnt = min(kNearTileF, nsrc - b0);
    __syncthreads();
    for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
      const int j = ib + b0 + q;
      float4 a = lpos[j], b = lnrm[j];
      const double A = (double)a.w;
      a.w = (float)(A * x[j]);
      b.w = (float)(A * x[n + j]);
      s_p[q] = a;
      s_l[q] = llo[j];
      s_n[q] = b;
    }
    __syncthreads();
    if (own) {
      const int self = t - (ib + b0);
#pragma unroll 4
      for (int q = 0; q < cnt; ++q) {
        const float4 a = s_p[q], l = s_l[q], b = s_n[q];
        const bool skip = (q == self);
        float dx = (a.x - tx) + (l.x - lx), dy = (a.y - ty) + (l.y - ly),
              dz = (a.z - tz) + (l.z - lz);
        if (skip) dx = 1.f;  // keeps the skipped pair finite
        float K1, K2, K3, K4;
        bie4(dx, dy, dz, vx, vy, vz, b.x, b.y, b.z, kappa, eps, inv_eps, K1, K2, K3, K4);
        const float w1 = skip ? 0.f : a.w, w2 = skip ? 0.f : b.w;
        p1 = fmaf(K1, w1, fmaf(K2, w2, p1));
        p2 = fmaf(K3, w1, fmaf(K4, w2, p2));
      }
    }
  }
  if (own) res[slot] = make_double2((double)p1, (double)p2);
}

__global__ void reduce_kernel(const int64_t* __restrict__ slot_off,
                              const double2* __restrict__ res, const double* __restrict__ x,
                              int n, int t0, int t1, double pre1, double pre2,
                              double* __restrict__ y) {
  int t = t0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= t1) return;
  double s1 = 0.0, s2 = 0.0;
  for (int64_t k = slot_off[t]; k < slot_off[t + 1]; ++k) {
    double2 r = res[k];
    s1 += r.x;
    s2 += r.y;
  }
  y[t] = pre1 * x[t] - s1;
  y[n + t] = pre2 * x[n + t] - s2;
}

template <int P>
void launch_moments(Handle& H, const double* x, bool f32, cudaStream_t s) {
  Tree& T = H.tree;
  if (T.nmslot == 0) return;
  const int nch = T.mslot_chunk0.back() + T.mslot_nchunk.back();
  if (f32) {
    auto partial = [&](auto sets) {
      constexpr int S = decltype(sets)::value;
      using M = MomShape<P, S>;
      TABI_K(K_MOMENTS, s);
      mom_partial_kernel<P, S><<<ceil_div(nch, M::CPB), M::G * M::CPB, 0, s>>>(
          T.d_mchunks.p, nch, T.d_mslot_node.p, T.d_mid.p, H.d_x.p, H.d_y.p, H.d_z.p, H.d_nx.p,
          H.d_ny.p, H.d_nz.p, H.d_area.p, x, H.n, H.d_mraw.p);
    };
    const bool few = (int64_t)H.n * tabi_nterms(P) <= kMomFew;
    if constexpr (P <= 5) {
      if (few) partial(std::integral_constant<int, 1>());
    }
    if (P > 5 || !few) partial(std::integral_constant<int, 4>());
    TABI_K(K_MOMENTS, s);
    mom_final_kernel<P><<<T.nmslot, 256, 0, s>>>(T.d_mslot_chunks.p, H.d_mraw.p, H.d_mwf.p);
    return;
  }
  if (harm_mom_smem(P) > 48 * 1024)
    raise_smem_limit((const void*)harm_mom_kernel<P>, harm_mom_smem(P));
  {
    TABI_K(K_MOMENTS, s);
    harm_mom_kernel<P><<<nch, 32 * harm_warps(P), harm_mom_smem(P), s>>>(
        T.d_mchunks.p, T.d_mslot_node.p, T.d_mid.p, H.d_x.p, H.d_y.p, H.d_z.p, H.d_nx.p,
        H.d_ny.p, H.d_nz.p, H.d_area.p, x, H.n, harm_beta<P>(H.prm.kappa),
        H.prm.eps1 / H.prm.eps0, H.d_mraw.p);
  }
  TABI_K(K_MOMENTS, s);
  harm_final_kernel<P><<<T.nmslot, 128, 0, s>>>(T.d_mslot_chunks.p, H.d_mraw.p, H.d_mw.p);
}

template <int P>
void launch_far(Handle& H, bool f32, cudaStream_t s) {
  Tree& T = H.tree;
  const int nw = (int)(T.ranged ? T.r_far_work.size() : T.far_work.size());
  const WorkItem* fw = T.ranged ? T.d_r_far_work.p : T.d_far_work.p;
  const int2* fe = T.ranged ? T.d_r_far_ent.p : T.d_far_ent.p;
  if (nw == 0) return;
  const double eps = H.prm.eps1 / H.prm.eps0;
  TABI_K(K_FAR, s);
  if (f32)
    far_kernel<P><<<nw, kFarThreads, 0, s>>>(
        fw, fe, H.d_mwf.p, T.d_mid.p, H.d_x.p, H.d_y.p, H.d_z.p,
        H.d_nx.p, H.d_ny.p, H.d_nz.p, (float)H.prm.kappa, (float)eps, H.d_res.p);
  else
    (T.far_nt > 1 ? far_harm_kernel<P, far_pair(P)> : far_harm_kernel<P, 1>)<<<
        nw, kFarThreads, 0, s>>>(fw, fe, H.d_mw.p, T.d_mid.p, H.d_x.p, H.d_y.p, H.d_z.p,
                                 H.d_nx.p, H.d_ny.p, H.d_nz.p, H.prm.kappa, 1.0 / eps,
                                 H.d_res.p);
}

// FP32 copies of the faces relative to their leaf centres (once per tree)
void prepare_f32(Handle& H, cudaStream_t s) {
  Tree& T = H.tree;
  if (T.lrel_ready) return;
  T.d_leaves.alloc(std::max(T.nleaf, 1));
  TABI_CUDA(cudaMemcpyAsync(T.d_leaves.p, T.leaves.data(), sizeof(int) * T.nleaf,
                            cudaMemcpyHostToDevice, s));
  T.d_lpos.alloc(std::max(H.n, 1));
  T.d_llo.alloc(std::max(H.n, 1));
  T.d_lnrm.alloc(std::max(H.n, 1));
  {
    TABI_K(K_TREE, s);
    leaf_rel_kernel<<<T.nleaf, 256, 0, s>>>(T.d_leaves.p, T.d_ibeg.p, T.d_num.p, T.d_mid.p,
                                            H.d_x.p, H.d_y.p, H.d_z.p, H.d_nx.p, H.d_ny.p,
                                            H.d_nz.p, H.d_area.p, T.d_lpos.p, T.d_llo.p,
                                            T.d_lnrm.p);
  }
  TABI_CUDA(cudaGetLastError());
  T.lrel_ready = true;
}

}  // namespace

double reduce_dev(Handle& H, int op, const double* a, const double* b, int n, cudaStream_t s) {
  H.d_red.alloc(kRedBlocks + 8);
  int nb = std::min(kRedBlocks, ceil_div(n, kRedThreads));
  if (nb < 1) nb = 1;
  if (op == 0)
    { TABI_K(K_VEC, s); reduce_partial_kernel<0><<<nb, kRedThreads, 0, s>>>(a, b, n, H.d_red.p); }
  else if (op == 1)
    { TABI_K(K_VEC, s); reduce_partial_kernel<1><<<nb, kRedThreads, 0, s>>>(a, b, n, H.d_red.p); }
  else
    { TABI_K(K_VEC, s); reduce_partial_kernel<2><<<nb, kRedThreads, 0, s>>>(a, b, n, H.d_red.p); }
  { TABI_K(K_VEC, s); reduce_final_kernel<<<1, 256, 0, s>>>(H.d_red.p, nb, H.d_red.p + kRedBlocks); }
  TABI_CUDA(cudaMemcpyAsync(H.h_pinned, H.d_red.p + kRedBlocks, sizeof(double),
                            cudaMemcpyDeviceToHost, s));
  TABI_CUDA(cudaStreamSynchronize(s));
  return H.h_pinned[0];
}

double asum_dev(Handle& H, const double* x, int n, cudaStream_t s) {
  return reduce_dev(H, 0, x, nullptr, n, s);
}
double dot_dev(Handle& H, const double* a, const double* b, int n, cudaStream_t s) {
  return reduce_dev(H, 1, a, b, n, s);
}
double nrm2_dev(Handle& H, const double* a, int n, cudaStream_t s) {
  return sqrt(reduce_dev(H, 2, a, nullptr, n, s));
}

void alloc_moments(Handle& H, int nchunk) {
  const int p = H.prm.order, nslot = H.tree.nmslot;
  const bool mixed = H.prm.precision == TABI_PREC_MIXED;
  H.d_mraw.alloc((size_t)nchunk * std::max(harm_raw(p), mixed ? 4 * tabi_nterms(p) : 0));
  H.d_mw.alloc((size_t)nslot * harm_size(p));
  if (mixed) H.d_mwf.alloc((size_t)nslot * 16 * tabi_nterms(p));
}

void matvec_dev(Handle& H, const double* x, double* y, cudaStream_t s, bool check_zero) {
  const int n = H.n;
  if (check_zero) {
    // MATVECmain (main.f90:478-479): sum|x| < 1e-10 gives y = x
    double a = asum_dev(H, x, 2 * n, s);
    if (a < 1e-10) {
      if (y != x)
        TABI_CUDA(cudaMemcpyAsync(y, x, sizeof(double) * 2 * n, cudaMemcpyDeviceToDevice, s));
      return;
    }
  }
  Tree& T = H.tree;
  const bool f32 = H.mv_prec == TABI_PREC_MIXED;
  if (f32) prepare_f32(H, s);
  TABI_PHASE(K_PHASE_MATVEC, s);
  // the near field runs on the handle's side stream, concurrently with the
  // moments + far field on s; both write disjoint result slots
  const int nnw = (int)(T.ranged ? T.r_near_work.size() : T.near_work.size());
  const WorkItem* nwk = T.ranged ? T.d_r_near_work.p : T.d_near_work.p;
  const int2* nent = T.ranged ? T.d_r_near_ent.p : T.d_near_ent.p;
  const bool fork = nnw > 0 && H.side != nullptr;
  cudaStream_t sn = fork ? H.side : s;
  if (fork) {
    TABI_CUDA(cudaEventRecord(H.ev_fork, s));
    TABI_CUDA(cudaStreamWaitEvent(sn, H.ev_fork, 0));
  }
  // moments first (small, needed by the far field), then the near field on
  // the side stream and the far field on s
  switch (H.prm.order) {
    case 1: launch_moments<1>(H, x, f32, s); break;
    case 2: launch_moments<2>(H, x, f32, s); break;
    case 3: launch_moments<3>(H, x, f32, s); break;
    case 4: launch_moments<4>(H, x, f32, s); break;
    case 5: launch_moments<5>(H, x, f32, s); break;
    case 6: launch_moments<6>(H, x, f32, s); break;
    case 7: launch_moments<7>(H, x, f32, s); break;
    case 8: launch_moments<8>(H, x, f32, s); break;
    default: throw Error(TABI_ERR_ARG, "order must be 1..8");
  }
  if (nnw > 0 && f32) {
    TABI_K(K_NEAR, sn);
    near_kernel_f32<<<nnw, kNearThreads, 0, sn>>>(
        nwk, nent, T.d_ibeg.p, T.d_num.p, T.d_mid.p, H.d_x.p, H.d_y.p,
        H.d_z.p, T.d_lpos.p, T.d_llo.p, T.d_lnrm.p, x, n, (float)H.prm.kappa,
        (float)(H.prm.eps1 / H.prm.eps0), H.d_res.p);
  } else if (nnw > 0) {
    TABI_K(K_NEAR, sn);
    auto launch = [&](auto* kernel) {
      kernel<<<nnw, kNearThreads, 0, sn>>>(
          nwk, nent, T.d_ibeg.p, T.d_num.p, T.d_mid.p, T.d_rad.p, H.d_x.p, H.d_y.p, H.d_z.p,
          H.d_nx.p, H.d_ny.p, H.d_nz.p, H.d_area.p, x, n, H.prm.kappa, H.prm.eps1 / H.prm.eps0, H.d_res.p);
    };
    switch (T.near_split) {
      case 1: launch(near_kernel<1>); break;
      case 2: launch(near_kernel<2>); break;
      case 4: launch(near_kernel<4>); break;
      case 8: launch(near_kernel<8>); break;
      default: launch(near_kernel<16>); break;
    }
  }
  switch (H.prm.order) {
    case 1: launch_far<1>(H, f32, s); break;
    case 2: launch_far<2>(H, f32, s); break;
    case 3: launch_far<3>(H, f32, s); break;
    case 4: launch_far<4>(H, f32, s); break;
    case 5: launch_far<5>(H, f32, s); break;
    case 6: launch_far<6>(H, f32, s); break;
    case 7: launch_far<7>(H, f32, s); break;
    case 8: launch_far<8>(H, f32, s); break;
    default: break;
  }
  if (fork) {
    TABI_CUDA(cudaEventRecord(H.ev_join, sn));
    TABI_CUDA(cudaStreamWaitEvent(s, H.ev_join, 0));
  }
  double eps = H.prm.eps1 / H.prm.eps0;
  const int t0 = T.ranged ? T.rt0 : 0, t1 = T.ranged ? T.rt1 : n;
  { TABI_K(K_REDUCE, s); reduce_kernel<<<ceil_div(t1 - t0, 256), 256, 0, s>>>(T.d_slot_off.p, H.d_res.p, x, n, t0, t1,
                                                 0.5 * (1.0 + eps), 0.5 * (1.0 + 1.0 / eps), y); }
  TABI_CUDA(cudaGetLastError());
}

namespace {

// FP64 direct sum of the operator for selected targets (the accuracy
// reference of the treecode): y_t = pre x_t - sum_{j != t} (K(t, j) A_j x_j),
// every source evaluated exactly (COMPP_DIRECT_PB's kernels,
// treecode3d_pb.f:919-1008).  Grid: x = chunks of kDirT targets (one per
// thread), y = chunks of kDirS sources staged through shared memory;
// partials per (target, source chunk) are summed in chunk order afterwards.
constexpr int kDirT = 128, kDirS = 8192, kDirTile = 256;

__global__ void __launch_bounds__(kDirT) direct_kernel(
    int n, const int* __restrict__ targets, int nt, const double* __restrict__ px,
    const double* __restrict__ py, const double* __restrict__ pz,
    const double* __restrict__ nx, const double* __restrict__ ny,
    const double* __restrict__ nz, const double* __restrict__ area,
    const double* __restrict__ x, double kappa, double eps, double2* __restrict__ part) {
  __shared__ double s_x[kDirTile], s_y[kDirTile], s_z[kDirTile];
  __shared__ double s_nx[kDirTile], s_ny[kDirTile], s_nz[kDirTile];
  __shared__ double s_w1[kDirTile], s_w2[kDirTile];
  const int k = blockIdx.x * kDirT + threadIdx.x;
  const bool own = k < nt;
  const int t = own ? targets[k] : 0;
  const double tx = px[t], ty = py[t], tz = pz[t], vx = nx[t], vy = ny[t], vz = nz[t];
  const double inv_eps = 1.0 / eps;
  const int j0 = blockIdx.y * kDirS, j1 = min(n, j0 + kDirS);
  double p1 = 0.0, p2 = 0.0;
  for (int b0 = j0; b0 < j1; b0 += kDirTile) {
    const int cnt = min(kDirTile, j1 - b0);
    __syncthreads();
    for (int q = threadIdx.x; q < cnt; q += kDirT) {
      const int j = b0 + q;
      s_x[q] = px[j];
      s_y[q] = py[j];
      s_z[q] = pz[j];
      s_nx[q] = nx[j];
      s_ny[q] = ny[j];
      s_nz[q] = nz[j];
      s_w1[q] = area[j] * x[j];
      s_w2[q] = area[j] * x[n + j];
    }
    __syncthreads();
    if (own)
      for (int q = 0; q < cnt; ++q) {
        const bool skip = (b0 + q == t);
        double dx = s_x[q] - tx, dy = s_y[q] - ty, dz = s_z[q] - tz;
        if (skip) dx = 1.0;
        double K1, K2, K3, K4;
        bie4<double>(dx, dy, dz, vx, vy, vz, s_nx[q], s_ny[q], s_nz[q], kappa, eps, inv_eps, K1,
                     K2, K3, K4);
        const double w1 = skip ? 0.0 : s_w1[q], w2 = skip ? 0.0 : s_w2[q];
        p1 = fma(K1, w1, fma(K2, w2, p1));
        p2 = fma(K3, w1, fma(K4, w2, p2));
      }
  }
  if (own) part[(size_t)k * gridDim.y + blockIdx.y] = make_double2(p1, p2);
}

__global__ void direct_final_kernel(int n, const int* __restrict__ targets, int nt, int nchunk,
                                    const double2* __restrict__ part,
                                    const double* __restrict__ x, double pre1, double pre2,
                                    double* __restrict__ y) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nt) return;
  const int t = targets[k];
  double s1 = 0.0, s2 = 0.0;
  for (int c = 0; c < nchunk; ++c) {
    const double2 r = part[(size_t)k * nchunk + c];
    s1 += r.x;
    s2 += r.y;
  }
  y[k] = pre1 * x[t] - s1;
  y[nt + k] = pre2 * x[n + t] - s2;
}

}  // namespace

void direct_targets_dev(Handle& H, int nt, const int* targets, const double* x, double* y,
                        cudaStream_t s) {
  TABI_REQUIRE(H.has_surface, TABI_ERR_STATE, "no surface");
  const int n = H.n;
  const int nchunk = ceil_div(n, kDirS);
  H.d_dirpart.alloc((size_t)std::max(nt, 1) * nchunk);
  const double eps = H.prm.eps1 / H.prm.eps0;
  {
    TABI_K(K_NEAR, s);
    direct_kernel<<<dim3(ceil_div(nt, kDirT), nchunk), kDirT, 0, s>>>(
        n, targets, nt, H.d_x.p, H.d_y.p, H.d_z.p, H.d_nx.p, H.d_ny.p, H.d_nz.p, H.d_area.p, x,
        H.prm.kappa, eps, H.d_dirpart.p);
  }
  {
    TABI_K(K_REDUCE, s);
    direct_final_kernel<<<ceil_div(nt, 256), 256, 0, s>>>(n, targets, nt, nchunk,
                                                          H.d_dirpart.p, x, 0.5 * (1.0 + eps),
                                                          0.5 * (1.0 + 1.0 / eps), y);
  }
  TABI_CUDA(cudaGetLastError());
}

void set_target_range(Handle& H, int t0, int t1, cudaStream_t s) {
  Tree& T = H.tree;
  const int n = H.n;
  TABI_REQUIRE(H.has_tree, TABI_ERR_STATE, "tabi_build_tree has not been called");
  TABI_REQUIRE(0 <= t0 && t0 < t1 && t1 <= n, TABI_ERR_ARG, "target range must be within 0..nface");
  T.ranged = false;
  if (t0 == 0 && t1 == n) return;
  // leaf-aligned: the shard owns whole leaves (so the preconditioner, which is
  // leaf-local, splits with it)
  std::vector<int> starts;
  for (int c : T.leaves) starts.push_back(T.ibeg[c]);
  std::sort(starts.begin(), starts.end());
  auto boundary = [&](int t) {
    return t == n || std::binary_search(starts.begin(), starts.end(), t);
  };
  TABI_REQUIRE(boundary(t0) && boundary(t1), TABI_ERR_ARG,
               "target range must start and end on leaf boundaries (tree order)");
  // the interaction entries of targets in range, item by item
  auto restrict_list = [&](const PinVec<WorkItem>& work, const DBuf<int2>& ent,
                           std::vector<WorkItem>& rwork, DBuf<WorkItem>& d_rwork,
                           DBuf<int2>& d_rent) {
    size_t total = 0;
    for (const WorkItem& w : work) total = std::max(total, (size_t)w.start + w.count);
    std::vector<int2> h(total), out;
    if (total)
      TABI_CUDA(cudaMemcpyAsync(h.data(), ent.p, sizeof(int2) * total, cudaMemcpyDeviceToHost,
                                s));
    TABI_CUDA(cudaStreamSynchronize(s));
    rwork.clear();
    for (const WorkItem& w : work) {
      const int start = (int)out.size();
      for (int k = 0; k < w.count; ++k) {
        const int2 e = h[(size_t)w.start + k];
        if (e.x >= t0 && e.x < t1) out.push_back(e);
      }
      const int cnt = (int)out.size() - start;
      if (cnt > 0) rwork.push_back(WorkItem{w.node, start, cnt, w.mslot});
    }
    d_rwork.alloc(std::max<size_t>(rwork.size(), 1));
    d_rent.alloc(std::max<size_t>(out.size(), 1));
    if (!rwork.empty())
      TABI_CUDA(cudaMemcpyAsync(d_rwork.p, rwork.data(), sizeof(WorkItem) * rwork.size(),
                                cudaMemcpyHostToDevice, s));
    if (!out.empty())
      TABI_CUDA(cudaMemcpyAsync(d_rent.p, out.data(), sizeof(int2) * out.size(),
                                cudaMemcpyHostToDevice, s));
  };
  restrict_list(T.far_work, T.d_far_ent, T.r_far_work, T.d_r_far_work, T.d_r_far_ent);
  restrict_list(T.near_work, T.d_near_ent, T.r_near_work, T.d_r_near_work, T.d_r_near_ent);
  // the preconditioner's leaves in range, in the apply's big / small classes
  std::vector<int> big, small;
  for (int l = 0; l < T.nleaf; ++l) {
    const int c = T.leaves[l], b0 = T.ibeg[c], nm = T.num[c];
    if (b0 >= t0 && b0 + nm <= t1) (2 * nm > kSolveSmall ? big : small).push_back(l);
  }
  auto by_size = [&](int a, int b) { return T.num[T.leaves[a]] > T.num[T.leaves[b]]; };
  std::sort(big.begin(), big.end(), by_size);
  std::sort(small.begin(), small.end(), by_size);
  T.r_solve_big = (int)big.size();
  T.r_solve_small = (int)small.size();
  big.insert(big.end(), small.begin(), small.end());
  T.d_r_solve_list.alloc(std::max<size_t>(big.size(), 1));
  if (!big.empty())
    TABI_CUDA(cudaMemcpyAsync(T.d_r_solve_list.p, big.data(), sizeof(int) * big.size(),
                              cudaMemcpyHostToDevice, s));
  TABI_CUDA(cudaStreamSynchronize(s));
  T.ranged = true;
  T.rt0 = t0;
  T.rt1 = t1;
}

}  // namespace tabi
