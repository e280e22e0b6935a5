// Rank-0 smooth PME (order-6 B-splines) on a cubic K^3 grid.
//
//   spread   : Q(g) = sum_i q_i M6(u_i,x) M6(u_i,y) M6(u_i,z)   (fixed-point or FP64 atomics)
//   R2C FFT  : S(k)
//   convolve : S(k) *= C(k)/theta(k)^2, E_rec = 1/2 sum_k C |S|^2/theta^2 (FP64, fixed order)
//   C2R FFT  : Phi(g)                                           (unnormalised)
//              these three by the plane kernels of pme_fft.cuh, or by cuFFT for the grid sides it
//              takes less time for (fft_planes)
//   gather   : phi_i = sum_g theta_i(g) Phi(g), dE/dx_i = q_i grad phi_i,
//              dE/dq_i = phi_i - 2 a q_i / sqrt(pi), E_self = -(a/sqrt(pi)) sum q^2
//
// Conventions follow the reference (torchff/pme_ref.py:11-469, csrc/pme/kernels.cuh):
// u = K * (box^-T r) per lattice direction, m0 = ceil(u), the 6 stencil points are
// m0-3 .. m0+2 with weights M6((m0 - u) + k), grid index gx*K^2 + gy*K + gz, and
// the signed frequency of FFT index i is i for 2i < K, else i - K.
#pragma once

#include <cufft.h>

#include "cluster.cuh"
#include "pme_fft.cuh"

namespace tff {

constexpr int kPmeBlock = 256;

struct PmeShared {
  double recip[9];
  double inv[9];
  double vol;
};

template <class T>
__device__ __forceinline__ void load_pme_shared(const T *box, int K, PmeShared &sh) {
  Box b;
  load_box(box, b);
  for (int d = 0; d < 3; ++d)
    for (int c = 0; c < 3; ++c) sh.recip[3 * d + c] = (double)K * b.inv[3 * c + d];
  for (int k = 0; k < 9; ++k) sh.inv[k] = b.inv[k];
  sh.vol = b.vol;
}

// Atom sources: caller order, or caller arrays in the order of a cluster build.
template <class T>
struct PlainAtoms {
  const T *x;
  const T *q;
  int64_t n;
  __device__ __forceinline__ bool get(int64_t t, double &rx, double &ry, double &rz, T &qi) const {
    if (t >= n) return false;
    rx = x[3 * t]; ry = x[3 * t + 1]; rz = x[3 * t + 2];
    qi = q[t];
    return true;
  }
};

// Atoms in the cluster (Hilbert) order of a cluster build: slot t is caller atom sidx[t]
// (-1: padding). Coordinates and charges come from the caller arrays, so every atom's
// numbers are those of PlainAtoms; only the visiting order changes, and neighbouring
// threads then touch neighbouring grid points.
template <class T>
struct IndexedAtoms {
  const T *x;
  const T *q;
  const int *sidx;
  int64_t n;  // slots
  __device__ __forceinline__ bool get(int64_t t, double &rx, double &ry, double &rz, T &qi) const {
    if (t >= n) return false;
    const int64_t a = sidx[t];
    if (a < 0) return false;
    rx = x[3 * a]; ry = x[3 * a + 1]; rz = x[3 * a + 2];
    qi = q[a];
    return true;
  }
};

// Stencils are computed by a warp for up to kStencilAtoms atoms at a time, one (atom, axis) per
// lane, into shared memory: the lanes that work on an atom then read its weights instead of
// evaluating the same splines each.
constexpr int kStencilAtoms = 10;

// One stencil point of an axis: weight and element offset of its index in the K^3 grid (the
// index, wrapped into [0, K), times the axis's stride). Entries are vector-aligned for one load.
template <class T> struct SplinePoint;
template <> struct __align__(8) SplinePoint<float> { float w; int off; };
template <> struct __align__(16) SplinePoint<double> { double w; int off; };

// Weight and derivative.
template <class T> struct SplinePoint2;
template <> struct __align__(16) SplinePoint2<float> { float w, d; int off; };
template <> struct __align__(16) SplinePoint2<double> { double w, d; int off; };

template <class T>
struct SpreadStage { SplinePoint<T> p[kStencilAtoms][3][6]; };
// Spline argument and grid offsets of an atom on axis d: returns w (the weights are M6(w + k))
// and calls put(k, offset) for the 6 points. recip[d*3 + c] = K * inv[c][d]: u_d = sum_c
// recip[d][c] r_c. The first point is wrapped into [0, K) by compares for atoms within a box
// length of the primary cell (the common case), by a 64-bit remainder otherwise.
template <class F>
__device__ __forceinline__ double axis_points(double rx, double ry, double rz, const PmeShared &sh, int K, int d,
                                              F put) {
  const double u = sh.recip[3 * d] * rx + sh.recip[3 * d + 1] * ry + sh.recip[3 * d + 2] * rz;
  const double m0 = ceil(u);
  long long g = (long long)m0 - 3;
  if (g >= -K && g < 2 * (long long)K) {
    g += g < 0 ? K : 0;
    g -= g >= K ? K : 0;
  } else {
    g %= K;
    if (g < 0) g += K;
  }
  const int stride = d == 0 ? K * K : d == 1 ? K : 1;  // K <= 1024: offsets fit 32 bits
  int at = (int)g;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    put(k, at * stride);
    at = at + 1 == K ? 0 : at + 1;
  }
  return m0 - u;
}

// Spread of atoms [0, n) by the blocks bid of nblk. A warp takes its staged atoms one by one, six
// lanes along z and five (x, y) rows at a time, so that an atomic instruction touches runs of six
// consecutive grid points: 81 L2 sectors per atom, where lanes over the rows touched one for
// each of the 216 points. FP32 contributions are rounded to fixed point one by one (the weight
// of the x axis carries the charge and the scale, a power of two), so the grid does not depend
// on the order of the atoms.
//
// Bound by the SM's reduction throughput (about one sector per clock) and L2 atomics. Alone: 300,000
// atoms FP32 160 -> 126 us against groups of three atoms with a lane per row, 9,000 atoms 11.7 ->
// 8.7 us; 30,000 scattered charges FP64 46 -> 20 us, 9,000 atoms 16.5 -> 9.5 us.
template <class T, class Atoms>
__device__ __forceinline__ void spread_atoms(const Atoms &atoms, int64_t n, const PmeShared &sh, int K,
                                             typename Acc<T>::S *grid, int64_t bid, int64_t nblk,
                                             SpreadStage<T> &S) {
  const int lane = threadIdx.x & 31;
  const int64_t wg = (bid * blockDim.x + threadIdx.x) / kWarp;
  const int64_t nw = nblk * blockDim.x / kWarp;
  // as many atoms per pass as it takes for them to fill the warps
  const int apw = (int)min((int64_t)kStencilAtoms, max((int64_t)1, (n + nw - 1) / nw));
  const int r0 = lane / 6, c = lane - 6 * r0;
  for (int64_t base = wg * apw; base < n; base += nw * apw) {
    __syncwarp();  // every lane is done with the previous pass's stencils
    if (lane < 3 * apw) {
      const int k = lane / 3, d = lane - 3 * k;
      SplinePoint<T>(&p)[6] = S.p[k][d];
      double rx, ry, rz;
      T q;
      if (base + k < n && atoms.get(base + k, rx, ry, rz, q)) {
        const double w = axis_points(rx, ry, rz, sh, K, d, [&](int i, int off) { p[i].off = off; });
        T val[6], der[6];
        bspline6<T>((T)w, val, der);
        if (d == 0) {
          if (sizeof(T) == 4) q *= T(kFixScale);
#pragma unroll
          for (int i = 0; i < 6; ++i) val[i] = q * val[i];
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) p[i].w = val[i];
      } else {
        p[0].off = -1;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int k = 0; k < apw; ++k) {
      const auto &p = S.p[k];
      if (p[0][0].off < 0 || lane >= 30) continue;
      const SplinePoint<T> pz = p[2][c], py = p[1][r0];
      const auto add = [&](const SplinePoint<T> &x, const SplinePoint<T> &y) {
        const T v = (x.w * y.w) * pz.w;
        const int at = x.off + y.off + pz.off;
        if constexpr (sizeof(T) == 4)
          atomicAdd(&grid[at], (unsigned long long)__float2ll_rn(v));
        else
          atomicAdd(&grid[at], v);
      };
      // rows (a, r0) for y indices 0..4, then the six rows of y index 5
#pragma unroll
      for (int a = 0; a < 6; ++a) add(p[0][a], py);
      const SplinePoint<T> p5 = p[1][5];
      add(p[0][r0], p5);
      if (r0 == 0) add(p[0][5], p5);
    }
  }
}

template <class T, class Atoms>
__global__ void __launch_bounds__(kPmeBlock) pme_spread_kernel(Atoms atoms, int64_t n, const T *box, int K,
                                                               typename Acc<T>::S *grid) {
  __shared__ PmeShared sh;
  __shared__ SpreadStage<T> st[kPmeBlock / kWarp];
  if (threadIdx.x == 0) load_pme_shared(box, K, sh);
  __syncthreads();
  spread_atoms<T>(atoms, n, sh, K, grid, blockIdx.x, gridDim.x, st[threadIdx.x >> 5]);
}

// Blocks of a kernel that takes one atom (spread) or kGatherAtoms (gather) per warp at a time, up
// to a few waves.
inline int pme_blocks(int64_t warps) {
  const int64_t blocks = (warps * kWarp + kPmeBlock - 1) / kPmeBlock;
  return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, (int64_t)sm_count() * 8));
}

template <class T> struct CplxOf;
template <> struct CplxOf<float> { using type = cufftComplex; };
template <> struct CplxOf<double> { using type = cufftDoubleComplex; };

// Influence function C(k) / theta(k)^2 of a box, C(k) = 4 pi exp(-k^2 / 4 alpha^2) / (V k^2).
struct Influence {
  double inv[9], four_pi_over_v, inv4a2;
};

__device__ __forceinline__ void load_influence(const PmeShared &sh, double alpha, Influence &f) {
  for (int k = 0; k < 9; ++k) f.inv[k] = sh.inv[k];
  f.four_pi_over_v = 4.0 * 3.14159265358979323846 / sh.vol;
  f.inv4a2 = 1.0 / (4.0 * alpha * alpha);
}

template <class T>
__device__ __forceinline__ double influence(const Influence &f, int K, int ix, int iy, int iz, const T *xmod,
                                            const T *ymod, const T *zmod) {
  if (ix == 0 && iy == 0 && iz == 0) return 0.0;
  const double two_pi = 2.0 * 3.14159265358979323846;
  const double mx = (2 * ix < K) ? ix : ix - K;
  const double my = (2 * iy < K) ? iy : iy - K;
  const double mz = (2 * iz < K) ? iz : iz - K;
  // k_c = 2 pi sum_d m_d inv[c][d]
  const double kx = two_pi * (mx * f.inv[0] + my * f.inv[1] + mz * f.inv[2]);
  const double ky = two_pi * (mx * f.inv[3] + my * f.inv[4] + mz * f.inv[5]);
  const double kz = two_pi * (mx * f.inv[6] + my * f.inv[7] + mz * f.inv[8]);
  const double ksq = kx * kx + ky * ky + kz * kz;
  const double th = (double)xmod[ix] * (double)ymod[iy] * (double)zmod[iz];
  return f.four_pi_over_v * exp(-ksq * f.inv4a2) / (ksq * th * th);
}

// Gather output: caller arrays (caller order), plain stores (one thread per atom).
template <class T>
struct PlainGatherOut {
  T *phi;    // dE/dq (N), nullable
  T *grad;   // dE/dx (N,3), nullable
  __device__ __forceinline__ void put(int64_t t, double phi_t, double gx, double gy, double gz) const {
    if (phi) phi[t] = (T)phi_t;
    if (grad) {
      grad[3 * t] = (T)gx;
      grad[3 * t + 1] = (T)gy;
      grad[3 * t + 2] = (T)gz;
    }
  }
};

// Gather output for IndexedAtoms: slot t's values go to caller atom sidx[t].
template <class T>
struct IndexedGatherOut {
  T *phi;   // dE/dq (N), nullable
  T *grad;  // dE/dx (N,3), nullable
  const int *sidx;
  __device__ __forceinline__ void put(int64_t t, double phi_t, double gx, double gy, double gz) const {
    const int64_t a = sidx[t];
    if (phi) phi[a] = (T)phi_t;
    if (grad) {
      grad[3 * a] = (T)gx;
      grad[3 * a + 1] = (T)gy;
      grad[3 * a + 2] = (T)gz;
    }
  }
};

// Gather of atoms [0, n): phi and its gradient at every atom, sums of grid value times spline
// weights (FP64 beyond six products along x). Returns this thread's share of the self energy
// -(a/sqrt(pi)) sum q^2.
//
// The lanes are those of the spread: six along z and five (x, y) rows at a time, so that a load
// touches runs of six consecutive points (an x plane per lane touched 30 rows with every load). A lane
// sums its rows against the x and y weights, then multiplies by its z weights; the four sums of four atoms are
// reduce-scattered over the warp together, one shuffle per value instead of five. 9,000 atoms FP32
// 11.9 -> 9.9 us; an energy with gradients of 30,000 scattered charges in FP64 121 -> 112 us.
constexpr int kGatherAtoms = 4;
template <class T>
struct GatherStage { SplinePoint2<T> p[kGatherAtoms][3][6]; };

// One halving step of a reduce-scatter over lane bit o: keeps the half of v[0, n) that the lane's
// bit selects, with the partner's share added.
template <int n>
__device__ __forceinline__ void halve(double (&v)[4 * kGatherAtoms], int o, int lane) {
  const bool up = (lane & o) != 0;
#pragma unroll
  for (int k = 0; k < n / 2; ++k) {
    const double keep = up ? v[k + n / 2] : v[k], send = up ? v[k] : v[k + n / 2];
    v[k] = keep + __shfl_xor_sync(kFull, send, o);
  }
}

template <class T, class Atoms, class Out>
__device__ __forceinline__ double gather_atoms(const Atoms &atoms, int64_t n, const PmeShared &sh, int K,
                                               const T *Phi, double alpha, const Out &out, int64_t bid,
                                               int64_t nblk, GatherStage<T> &S) {
  const double a_rpi = alpha / 1.7724538509055160273;
  const int lane = threadIdx.x & 31;
  const int r0 = lane / 6, c = lane - 6 * r0;
  const int64_t wg = (bid * blockDim.x + threadIdx.x) / kWarp;
  const int64_t nw = nblk * blockDim.x / kWarp;
  double e = 0.0;
  for (int64_t base = wg * kGatherAtoms; base < n; base += nw * kGatherAtoms) {
    __syncwarp();  // every lane is done with the previous pass's stencils
    T q = T(0);    // lane 3 k + d: charge of staged atom k, if there is one
    bool has = false;
    if (lane < 3 * kGatherAtoms) {
      const int k = lane / 3, d = lane - 3 * k;
      double rx, ry, rz;
      has = base + k < n && atoms.get(base + k, rx, ry, rz, q);
      if (has) {
        SplinePoint2<T>(&p)[6] = S.p[k][d];
        const double w = axis_points(rx, ry, rz, sh, K, d, [&](int i, int off) { p[i].off = off; });
        T val[6], der[6];
        bspline6<T>((T)w, val, der);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          p[i].w = val[i];
          p[i].d = der[i];
        }
      }
    }
    const unsigned valid = __ballot_sync(kFull, has);
    __syncwarp();
    double v[4 * kGatherAtoms];  // phi and its three spline-argument derivatives of each atom
#pragma unroll
    for (int k = 0; k < kGatherAtoms; ++k) {
      double *o = v + 4 * k;
      o[0] = o[1] = o[2] = o[3] = 0.0;
      if (!((valid >> (3 * k)) & 1u) || lane >= 30) continue;
      const auto &p = S.p[k];
      const SplinePoint2<T> pz = p[2][c], py = p[1][r0], p5 = p[1][5], pr = p[0][r0];
      const T *at = Phi + pz.off;
      // rows (a, r0) for y indices 0..4, then the six rows of y index 5: six products along x in the
      // grid's precision, everything after them in FP64
      T sw = T(0), sd = T(0);
#pragma unroll
      for (int a = 0; a < 6; ++a) {
        const SplinePoint2<T> px = p[0][a];
        const T g = at[px.off + py.off];
        sw += px.w * g;
        sd += px.d * g;
      }
      const T gr = at[pr.off + p5.off];
      T s5w = pr.w * gr, s5d = pr.d * gr;
      if (r0 == 0) {
        const SplinePoint2<T> px = p[0][5];
        const T g = at[px.off + p5.off];
        s5w += px.w * g;
        s5d += px.d * g;
      }
      const double yw = py.w, yd = py.d, y5w = p5.w, y5d = p5.d, zw = pz.w, zd = pz.d;
      const double ww = yw * (double)sw + y5w * (double)s5w;
      o[0] = zw * ww;
      o[1] = zw * (yw * (double)sd + y5w * (double)s5d);
      o[2] = zw * (yd * (double)sw + y5d * (double)s5w);
      o[3] = zd * ww;
    }
    static_assert(kGatherAtoms == 4, "the lane bits below are for 16 values");
    halve<16>(v, 16, lane);
    halve<8>(v, 8, lane);
    halve<4>(v, 4, lane);
    halve<2>(v, 2, lane);
    const double sum = v[0] + __shfl_xor_sync(kFull, v[0], 1);  // value lane / 2 of the sixteen
    const int k = lane >> 3;
    const double du0 = __shfl_down_sync(kFull, sum, 2), du1 = __shfl_down_sync(kFull, sum, 4),
                 du2 = __shfl_down_sync(kFull, sum, 6);
    const T qk = __shfl_sync(kFull, q, 3 * k);
    if ((lane & 7) == 0 && ((valid >> (3 * k)) & 1u)) {
      // u_d = m0 - frac_d + const, so d(stencil u)/dr_c = -recip[d][c]
      const double qd = (double)qk;
      const double gxv = -qd * (du0 * sh.recip[0] + du1 * sh.recip[3] + du2 * sh.recip[6]);
      const double gyv = -qd * (du0 * sh.recip[1] + du1 * sh.recip[4] + du2 * sh.recip[7]);
      const double gzv = -qd * (du0 * sh.recip[2] + du1 * sh.recip[5] + du2 * sh.recip[8]);
      out.put(base + k, sum - 2.0 * a_rpi * qd, gxv, gyv, gzv);
      e -= a_rpi * qd * qd;
    }
  }
  return e;
}

template <class T, class Atoms, class Out>
__global__ void __launch_bounds__(kPmeBlock) pme_gather_kernel(Atoms atoms, int64_t nthreads, const T *box, int K,
                                                               const T *Phi, double alpha, Out out, double *partials,
                                                               unsigned *ticket, double *e_self, const double *e_rec,
                                                               double e_scale, T *energy_out) {
  __shared__ PmeShared sh;
  __shared__ GatherStage<T> st[kPmeBlock / kWarp];
  if (threadIdx.x == 0) load_pme_shared(box, K, sh);
  __syncthreads();
  const double e = gather_atoms<T>(atoms, nthreads, sh, K, Phi, alpha, out, blockIdx.x, gridDim.x,
                                   st[threadIdx.x >> 5]);
  const bool last = grid_sum<kPmeBlock>(e, partials, ticket, e_self, false);
  if (last && threadIdx.x == 0 && energy_out) energy_out[0] = (T)(e_scale * (*e_rec + *e_self));
}

// ---- second derivatives along a coordinate direction u (force matching)
// With theta_i(g) the stencil weight and w_d = m0_d - u_d its spline argument
// (dw_d/dr_c = -recip[d][c]), v_i = recip u_i, G_d = d theta / d w_d, H_de = d2 theta / dw_d dw_e:
//   P(g)   = sum_i q_i u_i . grad theta_i(g) = -sum_i q_i sum_d v_d G_d(g)
//   psi    = the same influence-function convolution of P as Phi of Q
//   d/dx_i (sum_j u_j . dE/dx_j) = q_i recip^T (A v_i - B),  A_de = sum_g Phi H_de, B_d = sum_g psi G_d
//   d/dq_i (sum_j u_j . dE/dx_j) = -v_i . C + sum_g psi theta_i,  C_d = sum_g Phi G_d
// (the reciprocal energy is 1/2 Q.Phi; the self term has no coordinate dependence).
// Staging and lanes as in spread_atoms; the products are FP64 in both precisions.
struct DirStage {
  SplinePoint2<double> p[kStencilAtoms][3][6];
  double v[kStencilAtoms][3], q[kStencilAtoms];
};

template <class T>
__global__ void __launch_bounds__(kPmeBlock) pme_spread_dir_kernel(PlainAtoms<T> atoms, const T *dir, int64_t n,
                                                                   const T *box, int K, typename Acc<T>::S *grid) {
  __shared__ PmeShared sh;
  __shared__ DirStage st[kPmeBlock / kWarp];
  if (threadIdx.x == 0) load_pme_shared(box, K, sh);
  __syncthreads();
  DirStage &S = st[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t wg = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int64_t nw = (int64_t)gridDim.x * blockDim.x / kWarp;
  const int apw = (int)min((int64_t)kStencilAtoms, max((int64_t)1, (n + nw - 1) / nw));
  const int r0 = lane / 6, c = lane - 6 * r0;
  for (int64_t base = wg * apw; base < n; base += nw * apw) {
    __syncwarp();
    const int left = (int)min((int64_t)apw, n - base);
    if (lane < 3 * left) {
      const int k = lane / 3, d = lane - 3 * k;
      const int64_t t = base + k;
      double rx, ry, rz;
      T q;
      atoms.get(t, rx, ry, rz, q);
      const double ux = dir[3 * t], uy = dir[3 * t + 1], uz = dir[3 * t + 2];
      S.v[k][d] = sh.recip[3 * d] * ux + sh.recip[3 * d + 1] * uy + sh.recip[3 * d + 2] * uz;
      if (d == 0) S.q[k] = (double)q;
      SplinePoint2<double>(&p)[6] = S.p[k][d];
      const double w = axis_points(rx, ry, rz, sh, K, d, [&](int i, int off) { p[i].off = off; });
      T val[6], der[6];
      bspline6<T>((T)w, val, der);
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        p[i].w = (double)val[i];
        p[i].d = (double)der[i];
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int k = 0; k < left; ++k) {
      if (lane >= 30) continue;
      const auto &p = S.p[k];
      const double v0 = S.v[k][0], v1 = S.v[k][1], v2 = S.v[k][2], nq = -S.q[k];
      const SplinePoint2<double> pz = p[2][c], py = p[1][r0];
      const auto add = [&](const SplinePoint2<double> &x, const SplinePoint2<double> &y) {
        const double c_val = nq * (v0 * x.d * y.w + v1 * x.w * y.d);  // times val_z
        const double c_der = nq * v2 * x.w * y.w;                      // times der_z
        Acc<T>::add(&grid[x.off + y.off + pz.off], c_val * pz.w + c_der * pz.d);
      };
#pragma unroll
      for (int a = 0; a < 6; ++a) add(p[0][a], py);
      const SplinePoint2<double> p5 = p[1][5];
      add(p[0][r0], p5);
      if (r0 == 0) add(p[0][5], p5);
    }
  }
}

// Per atom: kc * d/dx_i and kc * d/dq_i of sum_j u_j . dE_rec/dx_j (kLanesPerAtom lanes per atom,
// lane g of them the (x, y) rows g, g + kLanesPerAtom, ...).
constexpr int kLanesPerAtom = 8;
constexpr int kAtomsPerWarp = kWarp / kLanesPerAtom;

template <class T>
__global__ void __launch_bounds__(kPmeBlock) pme_gather_hvp_kernel(PlainAtoms<T> atoms, const T *dir, int64_t n,
                                                                   const T *box, int K, const T *Phi, const T *Psi,
                                                                   double kc, T *hx, T *hq) {
  __shared__ PmeShared sh;
  if (threadIdx.x == 0) load_pme_shared(box, K, sh);
  __syncthreads();
  const int g = threadIdx.x % kLanesPerAtom;
  const int64_t wglob = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int64_t nwarps = (int64_t)gridDim.x * blockDim.x / kWarp;
  for (int64_t wb = wglob * kAtomsPerWarp; wb < n; wb += nwarps * kAtomsPerWarp) {
    const int64_t t = wb + (threadIdx.x % kWarp) / kLanesPerAtom;
    double rx = 0.0, ry = 0.0, rz = 0.0;
    T q = T(0);
    const bool ok = t < n && atoms.get(t, rx, ry, rz, q);
    // A00 A11 A22 A01 A02 A12, B0..2, C0..2, Psi_i
    double acc[13];
#pragma unroll
    for (int k = 0; k < 13; ++k) acc[k] = 0.0;
    T val[3][6], der[3][6], dd[3][6];
    int g0[3];
    if (ok) {
      const double r[3] = {rx, ry, rz};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double u = sh.recip[3 * d] * r[0] + sh.recip[3 * d + 1] * r[1] + sh.recip[3 * d + 2] * r[2];
        const double m0 = ceil(u);
        bspline6_d2<T>((T)(m0 - u), val[d], der[d], dd[d]);
        long long gg = (long long)m0 - 3;
        gg %= K;
        if (gg < 0) gg += K;
        g0[d] = (int)gg;
      }
      for (int rr = g; rr < 36; rr += kLanesPerAtom) {
        const int a = rr / 6, b = rr % 6;
        int gx = g0[0] + a, gy = g0[1] + b;
        gx -= (gx >= K) ? K : 0;
        gy -= (gy >= K) ? K : 0;
        const int64_t row = ((int64_t)gx * K + gy) * K;
        int gz = g0[2];
        double pv = 0.0, pd = 0.0, pdd = 0.0, sv = 0.0, sd = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const double ph = Phi[row + gz], ps = Psi[row + gz];
          pv += ph * (double)val[2][c];
          pd += ph * (double)der[2][c];
          pdd += ph * (double)dd[2][c];
          sv += ps * (double)val[2][c];
          sd += ps * (double)der[2][c];
          gz = (gz + 1 == K) ? 0 : gz + 1;
        }
        const double vx = val[0][a], dx = der[0][a], ddx = dd[0][a];
        const double vy = val[1][b], dy = der[1][b], ddy = dd[1][b];
        acc[0] += ddx * vy * pv;
        acc[1] += vx * ddy * pv;
        acc[2] += vx * vy * pdd;
        acc[3] += dx * dy * pv;
        acc[4] += dx * vy * pd;
        acc[5] += vx * dy * pd;
        acc[6] += dx * vy * sv;
        acc[7] += vx * dy * sv;
        acc[8] += vx * vy * sd;
        acc[9] += dx * vy * pv;
        acc[10] += vx * dy * pv;
        acc[11] += vx * vy * pd;
        acc[12] += vx * vy * sv;
      }
    }
#pragma unroll
    for (int k = 0; k < 13; ++k)
#pragma unroll
      for (int o = kLanesPerAtom / 2; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(kFull, acc[k], o);
    if (ok && g == 0) {
      const double ux = dir[3 * t], uy = dir[3 * t + 1], uz = dir[3 * t + 2];
      double v[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) v[d] = sh.recip[3 * d] * ux + sh.recip[3 * d + 1] * uy + sh.recip[3 * d + 2] * uz;
      const double A[3][3] = {{acc[0], acc[3], acc[4]}, {acc[3], acc[1], acc[5]}, {acc[4], acc[5], acc[2]}};
      double w[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) w[d] = A[d][0] * v[0] + A[d][1] * v[1] + A[d][2] * v[2] - acc[6 + d];
      const double qd = (double)q;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        hx[3 * t + c] = (T)(kc * qd * (sh.recip[c] * w[0] + sh.recip[3 + c] * w[1] + sh.recip[6 + c] * w[2]));
      hq[t] = (T)(kc * (-(v[0] * acc[9] + v[1] * acc[10] + v[2] * acc[11]) + acc[12]));
    }
  }
}

// ---- batched transforms: the plane kernels of pme_fft.cuh over every system of a batch. The work
// units are the planes of every grid (system s owns units plane_off .. plane_off + K - 1); the
// summation order of a plane is fixed, so a grid's result does not depend on the batch it runs in.
constexpr int kBatchFftThreads = 256;

// Next work unit of a persistent batched kernel, drawn from a per-launch counter (zeroed
// before the launch) so that blocks that finish early take more: returns the unit, equal
// to `units` or more when none is left. Called by every thread of the block; the first
// barrier also keeps the previous unit's shared memory until every thread is done with it.
__device__ __forceinline__ int next_unit(unsigned *counter) {
  __shared__ int s_unit;
  __syncthreads();
  if (threadIdx.x == 0) s_unit = (int)atomicAdd(counter, 1u);
  __syncthreads();
  return s_unit;
}

// The batch system owning work unit u: the largest s < nsys whose first unit (plane_off for
// transform planes, gather_off for gather and spread units) is at
// most u. Every system owns at least one unit of each kind.
enum BatchUnits { kUnitsPlanes = 0, kUnitsGather };
template <int KIND>
__device__ __forceinline__ int unit_system(const BatchSys *sys, int nsys, int u) {
  int lo = 0, hi = nsys - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const int off = KIND == kUnitsPlanes ? sys[mid].plane_off : sys[mid].gather_off;
    if (off <= u)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Persistent kernels over work units numbered across the batch: the planes of every grid, and
// units of a system's atoms for the spread and the gather (system s owns gather_off .. gather_off +
// gather_blocks - 1). A unit count depends on the system alone, so that its reductions sum in the
// same order whatever else is in the batch. Most blocks of a system's reductions:
constexpr int kBatchPmeMaxBlocks = 256;

enum BatchFftPass { kFftForward = 0, kFftSolve, kFftInverse };

template <class T, int PASS>
__device__ __forceinline__ void batch_fft_unit(const BatchSys &b, int sy, int p, typename Acc<T>::S *grid, T *real,
                                               Cplx<T> *cplx, const Cplx<T> *tables, const T *boxes, double alpha,
                                               const T *moduli, double *partials, unsigned *tickets, double *energies,
                                               PmeShared &sh, Influence &inf) {
  const int K = b.K, Kz = K / 2 + 1;
  FftPlan f = fft_plan<T>(K, tables + b.table_off);
  Cplx<T> *spec = cplx + b.cplx_off;
  const auto nothing = [] {};
  if constexpr (PASS == kFftForward) {
    fft_forward_plane<T>(f, grid + b.grid_off + (int64_t)p * K * K, spec + (int64_t)p * K * Kz, nothing);
  } else if constexpr (PASS == kFftInverse) {
    fft_inverse_plane<T>(f, spec + (int64_t)p * K * Kz, real + b.grid_off + (int64_t)p * K * K, nothing);
  } else {
    if (threadIdx.x == 0) {
      load_pme_shared(boxes + 9 * (int64_t)sy, K, sh);
      load_influence(sh, alpha, inf);
    }
    __syncthreads();
    const T *xm = moduli + b.mod_off, *ym = xm + K, *zm = ym + K;
    const double e = fft_solve_row<T>(
        f, spec, p, 0, Kz, [&](int ix, int iz) { return influence<T>(inf, K, ix, p, iz, xm, ym, zm); }, nothing, nothing);
    grid_sum_n<kBatchFftThreads>(0.5 * e, partials + (int64_t)kBatchPmeMaxBlocks * sy, tickets + 2 * sy,
                                 energies + 2 * sy, false, p, K);
  }
}

// partials: kBatchPmeMaxBlocks per system; tickets and energies: 2 per system
// ([2s] reciprocal, [2s+1] self).
template <class T, int PASS>
__global__ void __launch_bounds__(kBatchFftThreads, sizeof(T) == 4 ? 3 : 2)
    batch_fft_kernel(const BatchSys *sys, const BatchShape *shape, typename Acc<T>::S *grid, T *real, Cplx<T> *cplx,
                     const Cplx<T> *tables, const T *boxes, double alpha, const T *moduli, double *partials,
                     unsigned *tickets, double *energies, unsigned *counter) {
  __shared__ PmeShared sh;
  __shared__ Influence inf;
  const int nsys = shape->nsys, units = shape->plane_units;
  for (int u = next_unit(counter); u < units; u = next_unit(counter)) {
    const int sy = unit_system<kUnitsPlanes>(sys, nsys, u);
    batch_fft_unit<T, PASS>(sys[sy], sy, u - sys[sy].plane_off, grid, real, cplx, tables, boxes, alpha, moduli, partials,
                            tickets, energies, sh, inf);
  }
}

template <class S>
__global__ void batch_zero_grid_kernel(const BatchShape *shape, S *grid) {
  const int64_t n = shape->total_grid;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    grid[k] = 0;
}

// One PME block of one system (a separate call: the unit loop's state then does not share
// the inner loops' register allocation).
template <class T>
__device__ __noinline__ void batch_spread_unit(const BatchSys *sys, const T *x, const T *q, const T *boxes,
                                               typename Acc<T>::S *grid, int sy, int bx, PmeShared &sh,
                                               SpreadStage<T> &st) {
  const BatchSys &b = sys[sy];
  if (threadIdx.x == 0) load_pme_shared(boxes + 9 * (int64_t)sy, b.K, sh);
  __syncthreads();
  PlainAtoms<T> atoms{x + 3 * b.atom_off, q + b.atom_off, b.natoms};
  spread_atoms<T>(atoms, b.natoms, sh, b.K, grid + b.grid_off, bx, b.gather_blocks, st);
}

template <class T>
__global__ void __launch_bounds__(kPmeBlock, 4) batch_spread_kernel(const BatchSys *sys, const BatchShape *shape,
                                                                 const T *x, const T *q, const T *boxes,
                                                                 typename Acc<T>::S *grid, unsigned *counter) {
  __shared__ PmeShared sh;
  __shared__ SpreadStage<T> st[kPmeBlock / kWarp];
  // the gather's units (a system's atoms never outnumber its sorted slots)
  const int nsys = shape->nsys, units = shape->gather_units;
  for (int u = next_unit(counter); u < units; u = next_unit(counter)) {
    const int sy = unit_system<kUnitsGather>(sys, nsys, u);
    batch_spread_unit<T>(sys, x, q, boxes, grid, sy, u - sys[sy].gather_off, sh, st[threadIdx.x >> 5]);
  }
}

template <class T>
// The atoms of a system are visited in the cluster order of the batch's sort (sidx: sorted
// slot -> batch atom index, -1 for padding), so that neighbouring threads read neighbouring
// grid points; each atom's numbers are those of the caller-order visit.
__global__ void __launch_bounds__(kPmeBlock, sizeof(T) == 4 ? 3 : 2) batch_gather_kernel(const BatchSys *sys, const BatchShape *shape,
                                                                 const T *x, const T *q, const int *sidx,
                                                                 const T *boxes, const T *Phi, double alpha, T *phi,
                                                                 T *grad, double *partials, unsigned *tickets,
                                                                 double *energies, unsigned *counter) {
  __shared__ PmeShared sh;
  __shared__ GatherStage<T> st[kPmeBlock / kWarp];
  const int nsys = shape->nsys, units = shape->gather_units;
  for (int u = next_unit(counter); u < units; u = next_unit(counter)) {
    const int sy = unit_system<kUnitsGather>(sys, nsys, u);
    const BatchSys &b = sys[sy];
    const int bx = u - b.gather_off;
    if (threadIdx.x == 0) load_pme_shared(boxes + 9 * (int64_t)sy, b.K, sh);
    __syncthreads();
    const int *slots = sidx + b.cl_off * kWarp;
    const int64_t nslots = b.ncl * kWarp;
    IndexedAtoms<T> atoms{x, q, slots, nslots};
    IndexedGatherOut<T> out{phi, grad, slots};
    const double e = gather_atoms<T>(atoms, nslots, sh, b.K, Phi + b.grid_off, alpha, out, bx, b.gather_blocks,
                                     st[threadIdx.x >> 5]);
    grid_sum_n<kPmeBlock>(e, partials + (int64_t)kBatchPmeMaxBlocks * sy, tickets + 2 * sy + 1,
                          energies + 2 * sy + 1, false, bx, b.gather_blocks);
  }
}

// Scratch layout of one PME evaluation.
struct PmeLayout {
  int K;
  int64_t ngrid, ncplx;
  size_t fix, real, cplx, partials, tickets, energies, bytes;
  size_t zero_off, zero_bytes;
};

inline PmeLayout pme_layout(int dtype, int K) {
  PmeLayout L{};
  L.K = K;
  L.ngrid = (int64_t)K * K * K;
  L.ncplx = (int64_t)K * K * (K / 2 + 1);
  const size_t ts = dtype == TFF_F64 ? 8 : 4;
  Carver c(nullptr);
  // zeroed on every evaluation: reduction tickets, energies, the accumulation grid
  L.tickets = c.off; c.take<unsigned>(64);
  L.energies = (c.off + 255) & ~size_t(255); c.take<double>(8);
  L.fix = (c.off + 255) & ~size_t(255); c.take<char>(L.ngrid * 8);  // u64 fixed point (mixed) / double (FP64)
  L.zero_off = 0;
  L.zero_bytes = c.bytes();
  L.real = (c.off + 255) & ~size_t(255); c.take<char>(dtype == TFF_F64 ? 0 : L.ngrid * ts);
  L.cplx = (c.off + 255) & ~size_t(255); c.take<char>(L.ncplx * 2 * ts);
  L.partials = (c.off + 255) & ~size_t(255); c.take<double>(8192);
  L.bytes = c.bytes();
  return L;
}

struct PmePlanImpl {
  int dtype;
  int K;
  int device;
  bool planes;              // solved by the plane kernels (pme_fft.cuh), else by cuFFT
  void *tables = nullptr;   // planes: the tables of side K (fft_table)
  cufftHandle r2c, c2r;     // cuFFT plans otherwise
};

int pme_cufft_fail(cufftResult r, const char *what);

}  // namespace tff

struct tff_pme_plan_s {
  tff::PmePlanImpl impl;
};

namespace tff {

// FFT -> convolve -> FFT of the spread grid in ws (L.fix) on `s`; leaves the potential grid
// Phi in (T*)(ws + L.real) (mixed) or (T*)(ws + L.fix) (FP64), returned through *phi_grid.
// after_kernel: the work before it on the stream is a kernel. Defined in pme.cu.
template <class T>
int pme_solve_phase(const PmePlanImpl &p, const PmeLayout &L, char *ws, const T *box, double alpha, const T *xmod,
                    const T *ymod, const T *zmod, cudaStream_t s, T **phi_grid, bool after_kernel = true);

// Enqueue spread -> FFT -> convolve -> FFT on `s` (see pme_solve_phase for the result).
template <class T, class Atoms>
int pme_grid_phase(const PmePlanImpl &p, const PmeLayout &L, char *ws, Atoms atoms, int64_t nthreads, const T *box,
                   double alpha, const T *xmod, const T *ymod, const T *zmod, cudaStream_t s, T **phi_grid) {
  using S = typename Acc<T>::S;
  TFF_CUDA(cudaMemsetAsync(ws + L.zero_off, 0, L.zero_bytes, s));
  S *grid = reinterpret_cast<S *>(ws + L.fix);
  if (nthreads > 0) {
    pme_spread_kernel<T, Atoms><<<pme_blocks(nthreads), kPmeBlock, 0, s>>>(atoms, nthreads, box, p.K, grid);
    TFF_LAUNCHED();
  }
  return pme_solve_phase<T>(p, L, ws, box, alpha, xmod, ymod, zmod, s, phi_grid, nthreads > 0);
}

template <class T, class Atoms, class Out>
int pme_gather_phase(const PmePlanImpl &p, const PmeLayout &L, char *ws, Atoms atoms, int64_t nthreads, const T *box,
                     double alpha, const T *phi_grid, Out out, double e_scale, T *energy_out, cudaStream_t s) {
  double *partials = reinterpret_cast<double *>(ws + L.partials);
  unsigned *tickets = reinterpret_cast<unsigned *>(ws + L.tickets);
  double *energies = reinterpret_cast<double *>(ws + L.energies);
  const int nb = pme_blocks((nthreads + kGatherAtoms - 1) / kGatherAtoms);
  pme_gather_kernel<T, Atoms, Out><<<nb, kPmeBlock, 0, s>>>(atoms, nthreads, box, p.K, phi_grid, alpha, out,
                                                            partials, tickets + 1, energies + 1, energies, e_scale,
                                                            energy_out);
  TFF_LAUNCHED();
  return TFF_OK;
}

}  // namespace tff
