// Fused real-space kernels shared by the single-system and the batched evaluation.
//
// Tile kernel: one warp per work item = cluster I (lane l owns atom l of I) and up to
// kItemTiles clusters J taken with a stride from I's FULL neighbour list (entries k,
// k + n, k + 2n, ... for n = ceil(count / kItemTiles)), so that each item samples
// neighbours in every direction and the lanes get similar amounts of work.
//   pass 1: the J clusters are staged in shared memory; every lane sweeps the 32 atoms of
//           each with broadcast reads and builds a 32-bit in-cutoff mask per tile;
//   pass 2: each lane walks its own set bits across all tiles of the item and evaluates
//           LJ + erfc Coulomb only there;
//   pass 3: excluded pairs inside the cutoff get the Ewald exclusion correction.
// A cluster pair whose boxes are close enough uses one periodic shift for all its pairs
// (positions are cluster-contiguous images); other pairs use the per-pair minimum image.
// Each pair is evaluated from both sides, which removes j-side atomics: forces / charge
// gradients of atom i are summed in registers and added once per item into int64 fixed
// point accumulators (mixed) or FP64 atomics (FP64 mode); energies likewise, halved. With
// no block barrier a warp that finishes early does not wait for its block.
#pragma once

#include <cmath>
#include <vector>

#include "bonded.cuh"
#include "erf_poly.cuh"
#include "pme.cuh"

namespace tff {
namespace {


// Warps per block of the tile kernel: 4 (FP32) or 2 (FP64) so that the staged tiles fit in
// 48 KB of static shared memory.
// MODE 0: energy, dE/dx, dE/dq. MODE 1: also dE/dsigma and dE/d(sqrt eps). MODE 2: second
// derivatives along a coordinate direction u: d/dx, d/dq, d/dsigma, d/d(sqrt eps) of u . dE/dx.
template <class T, int MODE = 0> struct TileCfg {
  static constexpr int NW = (sizeof(T) == 8 || MODE == 2) ? 2 : 4;
};


__device__ __forceinline__ float erf_t(float x) { return erff(x); }
__device__ __forceinline__ double erf_t(double x) { return erf(x); }

// erfc(u) and exp(-u^2): libdevice in FP64, A&S 7.1.26 in FP32 (the MODE 0 FP32 path inlines
// the same approximation with paired instructions).
__device__ __forceinline__ void erfc_exp(double u, double &ec, double &ex) {
  ec = erfc(u);
  ex = exp(-u * u);
}
__device__ __forceinline__ void erfc_exp(float u, float &ec, float &ex) { erfc_exp_as(u, ec, ex); }
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt(x); }

template <class T>
struct TileArgs {
  ClusterData<T> cl;
  const typename V2<T>::type *lj;  // sorted slots: (sigma/2, sqrt(eps))
  const int *exslot;               // (npad, kMaxExcl) sorted slots of excluded partners, -1 padded
  typename Acc<T>::S *gx;          // (npad, 3) sorted slots, dE/dx
  typename Acc<T>::S *gq;          // (npad) sorted slots, dE/dq
  double rc, alpha, kc;
  typename Acc<T>::S *energies;    // per system: [2s] pairs (LJ + erfc Coulomb), [2s+1] exclusion correction
  typename Acc<T>::S *gs = nullptr;  // MODE 1/2: (npad) d/dsigma_i
  typename Acc<T>::S *ga = nullptr;  // MODE 1/2: (npad) d/da_i, a = sqrt(eps)
  const typename V4<T>::type *u = nullptr;  // MODE 2: direction per sorted slot
};

template <class T>
__device__ __forceinline__ void pair_min_image(bool ortho, T &dx, T &dy, T &dz, const T *m, const T *inv) {
  if (ortho) {
    dx = wrap1(dx, m[0], inv[0]);
    dy = wrap1(dy, m[4], inv[4]);
    dz = wrap1(dz, m[8], inv[8]);
  } else {
    min_image(dx, dy, dz, m, inv);
  }
}

// Resident 2-warp blocks per SM the register allocation of the FP64 energy kernel must allow: 10 (at
// most 96 registers). 3000 waters: 141 us per evaluation, 148 at 6, 149 at 13 (72 registers).
constexpr int kTileMinBlocks = 10;

// ERF (FP64): how the screened Coulomb terms are evaluated (erf_poly.cuh).
template <class T, int MODE = 0, int ERF = kErfLibrary>
__global__ void __launch_bounds__(TileCfg<T, MODE>::NW * 32, MODE == 0 ? kTileMinBlocks : 1)
    tile_kernel(TileArgs<T> A) {
  pdl_enter();
  using V = typename V4<T>::type;
  using W2 = typename V2<T>::type;
  constexpr int NW = TileCfg<T, MODE>::NW;
  __shared__ V s_pos[NW][kItemTiles][kWarp];
  __shared__ V s_u[NW][kItemTiles][MODE == 2 ? kWarp : 1];  // MODE 2: direction of the j atoms
  __shared__ W2 s_lj[NW][kItemTiles][kWarp];
  // negated j positions, structure of arrays, for the packed FP32 distance pass
  __shared__ __align__(16) float s_nx[NW][kItemTiles][sizeof(T) == 4 ? kWarp : 4];
  __shared__ __align__(16) float s_ny[NW][kItemTiles][sizeof(T) == 4 ? kWarp : 4];
  __shared__ __align__(16) float s_nz[NW][kItemTiles][sizeof(T) == 4 ? kWarp : 4];
  __shared__ unsigned s_mask[NW][kItemTiles][kWarp];   // in-cutoff, not excluded
  __shared__ unsigned s_xmask[NW][kItemTiles][kWarp];  // in-cutoff, excluded
  __shared__ int s_mi[NW][kItemTiles];                 // 1: tile needs the per-pair minimum image
  __shared__ T s_box[NW][2][9];                         // box and inverse of the warp's current system
  __shared__ T s_rpre2[NW];                             // squared j-atom prefilter radius of that system
  const ClusterData<T> &cl = A.cl;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T *s_m = s_box[w][0], *s_inv = s_box[w][1];
  int cur_sys = -1;
  bool ortho = false;
  const T rc2 = (T)(A.rc * A.rc);
  const float rc2_up = nextafterf((float)(A.rc * A.rc), INFINITY);  // FP32 pass 1: r2 <= rc2 <=> r2 < rc2_up
  const T alpha = (T)A.alpha;
  const T kc = (T)A.kc;
  const T two_a_rpi = (T)(2.0 * A.alpha / 1.7724538509055160273);
  const EwaldPoly<ERF == kErfLibrary ? kErfShort : ERF> ewald(A.alpha);  // unused with kErfLibrary

  const int nitems = cl.itemoff[cl.n_clusters()];
  const int nwarps = gridDim.x * NW;
  for (int it = blockIdx.x * NW + w; it < nitems; it += nwarps) {
    const int I = cl.items ? cl.items[it] : item_cluster(cl.itemoff, (int)cl.n_clusters(), it);
    const int isys = cl.system_of(I);
    if (isys != cur_sys) {
      const double *info = cl.info(isys);
      if (lane < 9) {
        s_m[lane] = (T)info[lane];
        s_inv[lane] = (T)info[9 + lane];
      }
      ortho = info[18] != 0.0;
      cur_sys = isys;
      if (lane == 0) {
        const T rpre = (T)(A.rc + 1e-3 + 1e-5 * (info[0] + info[4] + info[8]));
        s_rpre2[w] = rpre * rpre;
      }
      __syncwarp();
    }
    const int k = it - cl.itemoff[I];
    const int nch = cl.itemoff[I + 1] - cl.itemoff[I];
    const int cnt = cl.ncount[I];
    const int ntile = (cnt - k + nch - 1) / nch;  // this item takes list entries k, k+nch, ...
    const int64_t si = (int64_t)I * kWarp + lane;
    const bool vi = cl.sidx[si] >= 0;
    const V pi = cl.pos[si];
    const W2 lji = A.lj[si];
    const T kqi = kc * pi.w;
    const V ci = cl.bc[I], hi_ = cl.bh[I];
    V ui{};
    if constexpr (MODE == 2) ui = A.u[si];
    // Per-atom shift: every j atom is moved to its image nearest the centre c of cluster I.
    // If h + rc < L/2 on every axis (h: I's half extent), another image of j would be at
    // least L - rc away from an i atom while the chosen one is at most h + L/2 away, so every
    // pair within the cutoff gets its minimum-image displacement and no pair outside the
    // cutoff can appear inside it.
    const bool atom_shift = ortho && (hi_.x + (T)A.rc * s_inv[0] < T(0.499)) &&
                            (hi_.y + (T)A.rc * s_inv[4] < T(0.499)) && (hi_.z + (T)A.rc * s_inv[8] < T(0.499));
    const T cx = ci.x * s_m[0], cy = ci.y * s_m[4], cz = ci.z * s_m[8];

    // Excluded partners of atom i are sorted slots (-1: none), read per tile from two 16-byte
    // loads. Only tiles whose cluster J lies in the warp's range of partner clusters
    // [x_lo, x_hi] (warp-uniform) can hold an excluded pair; the others skip the check.
    const int4 *xs_row = reinterpret_cast<const int4 *>(A.exslot + si * kMaxExcl);
    int x_lo, x_hi;
    {
      const int4 a = xs_row[0], b = xs_row[1];
      const int xs[kMaxExcl] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      int lo = 0x7fffffff, hi = -1;
#pragma unroll
      for (int x = 0; x < kMaxExcl; ++x)
        if (xs[x] >= 0) {
          lo = min(lo, xs[x] >> 5);
          hi = max(hi, xs[x] >> 5);
        }
      x_lo = __reduce_min_sync(kFull, lo);
      x_hi = __reduce_max_sync(kFull, hi);
    }

    // stage the tiles and build their cutoff masks (pass 1)
    for (int t = 0; t < ntile; ++t) {
      const int J = cl.nbr[(int64_t)I * cl.cap + k + t * nch];
      const int64_t sj = (int64_t)J * kWarp + lane;
      // one periodic shift for the whole cluster pair when every pair's displacement then
      // lies within half a box length per axis (orthorhombic boxes)
      bool shifted = false;
      T sx = T(0), sy = T(0), sz = T(0);
      if (ortho && !atom_shift) {
        const V cj = cl.bc[J], hj = cl.bh[J];
        const T dcx = ci.x - cj.x, dcy = ci.y - cj.y, dcz = ci.z - cj.z;
        const T nx = floor(dcx + T(0.5)), ny = floor(dcy + T(0.5)), nz = floor(dcz + T(0.5));
        shifted = (fabs(dcx - nx) + hi_.x + hj.x < T(0.49)) && (fabs(dcy - ny) + hi_.y + hj.y < T(0.49)) &&
                  (fabs(dcz - nz) + hi_.z + hj.z < T(0.49));
        sx = nx * s_m[0];
        sy = ny * s_m[4];
        sz = nz * s_m[8];
      }
      V pj = cl.pos[sj];
      if (atom_shift) {
        pj.x += rint((cx - pj.x) * s_inv[0]) * s_m[0];
        pj.y += rint((cy - pj.y) * s_inv[4]) * s_m[4];
        pj.z += rint((cz - pj.z) * s_inv[8]) * s_m[8];
        shifted = true;
      } else if (shifted) {
        pj.x += sx;
        pj.y += sy;
        pj.z += sz;
      }
      bool keep_j = cl.sidx[sj] >= 0;
      if (shifted && J != I) {
        const T ex_ = fmax(fabs(pj.x - cx) - hi_.x * s_m[0], T(0)), ey_ = fmax(fabs(pj.y - cy) - hi_.y * s_m[4], T(0)),
                ez_ = fmax(fabs(pj.z - cz) - hi_.z * s_m[8], T(0));
        keep_j = keep_j && (ex_ * ex_ + ey_ * ey_ + ez_ * ez_ <= s_rpre2[w]);
      }
      const unsigned keep = __ballot_sync(kFull, keep_j);
      const unsigned lt_mask = lanemask_lt();
      const int nkeep = __popc(keep);
      const int n4 = (nkeep + 3) >> 2;
      if (keep_j) {
        const int slot = __popc(keep & lt_mask);
        s_pos[w][t][slot] = pj;
        s_lj[w][t][slot] = A.lj[sj];
        if constexpr (MODE == 2) s_u[w][t][slot] = A.u[sj];
        if (sizeof(T) == 4) {
          s_nx[w][t][slot] = -(float)pj.x;
          s_ny[w][t][slot] = -(float)pj.y;
          s_nz[w][t][slot] = -(float)pj.z;
        }
      }
      if (sizeof(T) == 4 && lane >= nkeep && lane < 4 * n4) {
        s_nx[w][t][lane] = 1e18f;
        s_ny[w][t][lane] = 1e18f;
        s_nz[w][t][lane] = 1e18f;
      }
      __syncwarp();
      unsigned mask = 0u;
      if (sizeof(T) == 4 && shifted) {
        // four j atoms per shared load, two per paired FP32 instruction (FADD2/FFMA2). The
        // FMA chain starts from -rc2' (rc2' = the float just above rc^2), so its result is
        // negative exactly for the pairs inside the cutoff and the sign bit is the mask bit:
        // a funnel shift appends it (first atom ends in bit 31; reversed once per tile).
        const float2 px = make_float2((float)pi.x, (float)pi.x), py = make_float2((float)pi.y, (float)pi.y),
                     pz = make_float2((float)pi.z, (float)pi.z);
        const float2 nrc2 = make_float2(-rc2_up, -rc2_up);
#pragma unroll
        for (int s = 0; s < kWarp; s += 4) {
          if (s >= 4 * n4) break;
          const float4 nx = *reinterpret_cast<const float4 *>(&s_nx[w][t][s]);
          const float4 ny = *reinterpret_cast<const float4 *>(&s_ny[w][t][s]);
          const float4 nz = *reinterpret_cast<const float4 *>(&s_nz[w][t][s]);
          float2 dx = __fadd2_rn(px, make_float2(nx.x, nx.y)), dy = __fadd2_rn(py, make_float2(ny.x, ny.y)),
                 dz = __fadd2_rn(pz, make_float2(nz.x, nz.y));
          float2 d2 = __ffma2_rn(dx, dx, nrc2);
          d2 = __ffma2_rn(dy, dy, d2);
          d2 = __ffma2_rn(dz, dz, d2);
          mask = __funnelshift_l(__float_as_uint(d2.x), mask, 1);
          mask = __funnelshift_l(__float_as_uint(d2.y), mask, 1);
          dx = __fadd2_rn(px, make_float2(nx.z, nx.w));
          dy = __fadd2_rn(py, make_float2(ny.z, ny.w));
          dz = __fadd2_rn(pz, make_float2(nz.z, nz.w));
          d2 = __ffma2_rn(dx, dx, nrc2);
          d2 = __ffma2_rn(dy, dy, d2);
          d2 = __ffma2_rn(dz, dz, d2);
          mask = __funnelshift_l(__float_as_uint(d2.x), mask, 1);
          mask = __funnelshift_l(__float_as_uint(d2.y), mask, 1);
        }
        mask = n4 > 0 ? __brev(mask) >> (kWarp - 4 * n4) : 0u;
      } else {
#pragma unroll 4
        for (int s = 0; s < nkeep; ++s) {
          const V q = s_pos[w][t][s];
          T dx = pi.x - q.x, dy = pi.y - q.y, dz = pi.z - q.z;
          if (!shifted) pair_min_image(ortho, dx, dy, dz, s_m, s_inv);
          const T r2 = dx * dx + dy * dy + dz * dz;
          mask |= (r2 <= rc2) ? (1u << s) : 0u;
        }
      }
      if (nkeep < kWarp) mask &= (1u << nkeep) - 1u;
      if (J == I) mask &= ~(1u << __popc(keep & lt_mask));
      if (!vi) mask = 0u;
      unsigned emask = 0u;
      if (J >= x_lo && J <= x_hi && mask) {
        const int4 a = xs_row[0], b = xs_row[1];
        const int xs[kMaxExcl] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int x = 0; x < kMaxExcl; ++x) {
          const int o = xs[x] & 31;
          if ((xs[x] >> 5) == J && ((keep >> o) & 1u)) emask |= 1u << __popc(keep & ((1u << o) - 1u));
        }
      }
      s_mask[w][t][lane] = mask & ~emask;
      s_xmask[w][t][lane] = mask & emask;
      if (lane == 0) s_mi[w][t] = !shifted;
    }
    __syncwarp();

    // pass 2: every lane walks its own in-cutoff pairs across all tiles of the item
    T fx = T(0), fy = T(0), fz = T(0), dq = T(0);
    double ep = 0.0;
    T d_sig = T(0), d_a = T(0);  // MODE 1/2: sigma and sqrt(eps) derivatives of atom i
    if constexpr (MODE != 0) {
      // one pair per step. With D = (dE/dr)/r of the pair: MODE 1 adds dE/dsigma_i and
      // dE/da_i; MODE 2 accumulates, with delta = u_i - u_j and rd = r_ij . delta,
      // d/dx_i (u . dE/dx) = D delta + (dD/dr / r) rd r_ij and the parameter derivatives
      // (dD/dp) rd (coordinates: fx..fz, charge: dq (times k later), sigma: d_sig, a: d_a)
      T te = T(0);
      int t = 0, iter = 0;
      unsigned m = ntile > 0 ? s_mask[w][0][lane] : 0u;
      while (true) {
        while (m == 0u && ++t < ntile) m = s_mask[w][t][lane];
        const bool have = m != 0u;
        if (!__any_sync(kFull, have)) break;
        if (MODE == 1 && (++iter & 15) == 0) {
          ep += (double)te;
          te = T(0);
        }
        if (have) {
          const int s = __ffs(m) - 1;
          m &= m - 1u;
          const V q = s_pos[w][t][s];
          const W2 ljj = s_lj[w][t][s];
          T dx = pi.x - q.x, dy = pi.y - q.y, dz = pi.z - q.z;
          if (s_mi[w][t]) pair_min_image(ortho, dx, dy, dz, s_m, s_inv);
          const T r2 = dx * dx + dy * dy + dz * dz;
          // f = erfc(alpha r) / r, g = -(1/r) df/dr, h = -(1/r) dg/dr (MODE 2)
          T rinv, rinv2, f, g, h = T(0);
          if constexpr (ERF != kErfLibrary) {
            rinv = rsqrt_t(r2);
            rinv2 = rcp_newton(r2, rinv);
            T tx;
            ewald.eval(r2, rinv, rinv2, f, g, tx);
            if constexpr (MODE == 2) h = ewald.second(rinv2, g, tx);
          } else {
            rinv = rsqrt_t(r2);
            rinv2 = rinv * rinv;
            const T u = alpha * (r2 * rinv);
            T ec, ex2;
            erfc_exp(u, ec, ex2);
            f = ec * rinv;
            g = (ec * rinv2 + two_a_rpi * ex2 * rinv) * rinv;
            if constexpr (MODE == 2) {
              const T rinv4 = rinv2 * rinv2;
              h = T(3) * ec * rinv4 * rinv + two_a_rpi * ex2 * (T(3) * rinv4 + T(2) * alpha * alpha * rinv2);
            }
          }
          const T sig = lji.x + ljj.x, aj = ljj.y, eps = lji.y * aj;
          const T sr = sig * rinv, sr2 = sr * sr, sr6 = sr2 * sr2 * sr2, sr12 = sr6 * sr6, s5 = sr2 * sr2 * sr;
          const T dcq = -q.w * g;  // D_coulomb / (k q_i)
          const T dlj = T(-24) * eps * (T(2) * sr12 - sr6) * rinv2;           // D_lj
          const T D = kqi * dcq + dlj;
          if constexpr (MODE == 1) {
            fx += D * dx;
            fy += D * dy;
            fz += D * dz;
            dq += q.w * f;
            te += kqi * q.w * f + T(4) * eps * (sr12 - sr6);
            d_sig += T(12) * eps * rinv * s5 * (T(2) * sr6 - T(1));  // 1/2 dE/dsigma_ij
            d_a += T(4) * aj * (sr12 - sr6);                       // dE/da_i
          } else {
            const V uj = s_u[w][t][s];
            const T ddx = ui.x - uj.x, ddy = ui.y - uj.y, ddz = ui.z - uj.z;
            const T rd = dx * ddx + dy * ddy + dz * ddz;
            const T rinv4 = rinv2 * rinv2;
            const T e2 = kqi * q.w * h +
                         T(24) * eps * (T(28) * sr12 - T(8) * sr6) * rinv4;  // (dD/dr) / r
            const T e2rd = e2 * rd;
            fx += D * ddx + e2rd * dx;
            fy += D * ddy + e2rd * dy;
            fz += D * ddz + e2rd * dz;
            dq += dcq * rd;
            d_sig += T(-72) * eps * rinv2 * rinv * s5 * (T(4) * sr6 - T(1)) * rd;  // 1/2 dD/dsigma_ij rd
            d_a += T(-24) * aj * (T(2) * sr12 - sr6) * rinv2 * rd;              // dD/da_i rd
          }
        }
      }
      ep += (double)te;
    } else {
      T te = T(0);  // partial energy, moved into ep every 16 pairs
      int t = 0, iter = 0;
      unsigned m = ntile > 0 ? s_mask[w][0][lane] : 0u;
      while (true) {
        while (m == 0u && ++t < ntile) m = s_mask[w][t][lane];
        const bool have = m != 0u;
        if (!__any_sync(kFull, have)) break;
        if ((++iter & 15) == 0) {
          ep += (double)te;
          te = T(0);
        }
        if (have) {
          const int s = __ffs(m) - 1;
          m &= m - 1u;
          const V q = s_pos[w][t][s];
          const W2 ljj = s_lj[w][t][s];
          T dx = pi.x - q.x, dy = pi.y - q.y, dz = pi.z - q.z;
          if (s_mi[w][t]) pair_min_image(ortho, dx, dy, dz, s_m, s_inv);
          const T r2 = dx * dx + dy * dy + dz * dz;
          T rinv, rinv2, f, g;
          if constexpr (ERF != kErfLibrary) {
            rinv = rsqrt_t(r2);
            rinv2 = rcp_newton(r2, rinv);
            T tx;
            ewald.eval(r2, rinv, rinv2, f, g, tx);
          } else {
            rinv = rsqrt_t(r2);
            rinv2 = rinv * rinv;
            const T u = alpha * (r2 * rinv);
            T ec, ex2;
            erfc_exp(u, ec, ex2);
            f = ec * rinv;
            g = (ec * rinv2 + two_a_rpi * ex2 * rinv) * rinv;
          }
          const T cq = q.w * f;  // E_coul / (k q_i)
          T dedr_r = -kqi * q.w * g;
          const T sig = lji.x + ljj.x;
          const T eps = lji.y * ljj.y;
          const T sr2 = sig * sig * rinv2;
          const T sr6 = sr2 * sr2 * sr2;
          dedr_r -= T(24) * eps * sr6 * (T(2) * sr6 - T(1)) * rinv2;
          fx += dedr_r * dx;
          fy += dedr_r * dy;
          fz += dedr_r * dz;
          dq += cq;
          te += kqi * cq + T(4) * eps * sr6 * (sr6 - T(1));
        }
      }
      ep += (double)te;
    }
    // pass 3: excluded pairs within the cutoff: Ewald exclusion correction
    // k q_i q_j (erfc(u) - 1)/r = -k q_i q_j erf(u)/r, no LJ
    double ex = 0.0;
    int t = 0;
    unsigned m = ntile > 0 ? s_xmask[w][0][lane] : 0u;
    while (true) {
      while (m == 0u && ++t < ntile) m = s_xmask[w][t][lane];
      const bool have = m != 0u;
      if (!__any_sync(kFull, have)) break;
      if (have) {
        const int s = __ffs(m) - 1;
        m &= m - 1u;
        const V q = s_pos[w][t][s];
        T dx = pi.x - q.x, dy = pi.y - q.y, dz = pi.z - q.z;
        if (s_mi[w][t]) pair_min_image(ortho, dx, dy, dz, s_m, s_inv);
        const T r2 = dx * dx + dy * dy + dz * dz;
        // f = -erf(alpha r) / r, g = -(1/r) df/dr, h = -(1/r) dg/dr (MODE 2)
        T f, g, h = T(0);
        if constexpr (ERF != kErfLibrary) {
          ewald.excluded(r2, f, g);
          if constexpr (MODE == 2) h = ewald.excluded_second(r2, g);
        } else {
          const T rinv = rsqrt_t(r2);
          const T u = alpha * (r2 * rinv);
          const T damp = -erf_t(u);
          const T ex2 = exp(-u * u);
          f = damp * rinv;
          g = (damp * rinv * rinv + two_a_rpi * ex2 * rinv) * rinv;
          if constexpr (MODE == 2) {
            const T rinv2 = rinv * rinv, rinv4 = rinv2 * rinv2;
            h = T(3) * damp * rinv4 * rinv + two_a_rpi * ex2 * (T(3) * rinv4 + T(2) * alpha * alpha * rinv2);
          }
        }
        const T cq = q.w * f;
        const T dcq = -q.w * g;
        const T dedr_r = kqi * dcq;
        if constexpr (MODE == 2) {
          // same form as the erfc term with erfc(u) -> erfc(u) - 1 (equal derivatives)
          const V uj = s_u[w][t][s];
          const T ddx = ui.x - uj.x, ddy = ui.y - uj.y, ddz = ui.z - uj.z;
          const T rd = dx * ddx + dy * ddy + dz * ddz;
          const T e2rd = kqi * q.w * h * rd;
          fx += dedr_r * ddx + e2rd * dx;
          fy += dedr_r * ddy + e2rd * dy;
          fz += dedr_r * ddz + e2rd * dz;
          dq += dcq * rd;
        } else {
          fx += dedr_r * dx;
          fy += dedr_r * dy;
          fz += dedr_r * dz;
          dq += cq;
          ex += (double)(kqi * cq);
        }
      }
    }
    if (vi) {
      Acc<T>::add(&A.gx[3 * si], (double)fx);
      Acc<T>::add(&A.gx[3 * si + 1], (double)fy);
      Acc<T>::add(&A.gx[3 * si + 2], (double)fz);
      Acc<T>::add(&A.gq[si], (double)kc * (double)dq);
      if constexpr (MODE != 0) {
        Acc<T>::add(&A.gs[si], (double)d_sig);
        Acc<T>::add(&A.ga[si], (double)d_a);
      }
    }
    // energies: warp sum, then one order-independent accumulation per work item
    ep = warp_sum(ep);
    ex = warp_sum(ex);
    if (MODE != 2 && lane == 0) {
      Acc<T>::add(&A.energies[2 * isys], 0.5 * ep);
      Acc<T>::add(&A.energies[2 * isys + 1], 0.5 * ex);
    }
    __syncwarp();
  }
}

// Sorted real-space accumulators + caller-order PME derivatives -> caller order; energies
// of each of the nsys systems (e_tile_acc and e_pme hold two values per system, terms
// gets four: real-space pairs, exclusion correction, reciprocal, self).
// With `bonded` (one system): its caller-order dE/dx (3N) and the bond and angle energies
// (at 3N, 3N + 1) are added too, and terms gets six values (+ bonds, angles).
template <class T>
__global__ void finalize_kernel(ClusterData<T> cl, const typename Acc<T>::S *gx, const typename Acc<T>::S *gq,
                                const T *pme_grad, const T *pme_phi, T *forces, double *forces64, T *grad_q,
                                const typename Acc<T>::S *e_tile_acc, const double *e_pme, double kc,
                                double *energy, double *terms, int nsys,
                                const typename Acc<T>::S *bonded = nullptr, unsigned *status_out = nullptr) {
  pdl_enter();
  // the build's overflow word (bit 0: a cluster's neighbour list was cut at its capacity),
  // copied out for a host caller that reads it together with the energy
  if (status_out && blockIdx.x == 0 && threadIdx.x == 0) *status_out = cl.status[0];
  const int64_t natoms = cl.n_atoms();
  if (cl.shape) nsys = cl.shape->nsys;
  for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < natoms;
       a += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = cl.inv[a];
    double x = Acc<T>::get(&gx[3 * s]), y = Acc<T>::get(&gx[3 * s + 1]), z = Acc<T>::get(&gx[3 * s + 2]);
    double g = Acc<T>::get(&gq[s]);
    if (bonded) {
      x += Acc<T>::get(&bonded[3 * a]);
      y += Acc<T>::get(&bonded[3 * a + 1]);
      z += Acc<T>::get(&bonded[3 * a + 2]);
    }
    if (pme_grad) {
      x += kc * (double)pme_grad[3 * a];
      y += kc * (double)pme_grad[3 * a + 1];
      z += kc * (double)pme_grad[3 * a + 2];
      g += kc * (double)pme_phi[a];
    }
    if (forces) {
      forces[3 * a] = (T)(-x);
      forces[3 * a + 1] = (T)(-y);
      forces[3 * a + 2] = (T)(-z);
    }
    if (forces64) {
      forces64[3 * a] = -x;
      forces64[3 * a + 1] = -y;
      forces64[3 * a + 2] = -z;
    }
    if (grad_q) grad_q[a] = (T)g;
  }
  for (int sy = blockIdx.x * blockDim.x + threadIdx.x; sy < nsys; sy += gridDim.x * blockDim.x) {
    const double e_tile[2] = {Acc<T>::get(&e_tile_acc[2 * sy]), Acc<T>::get(&e_tile_acc[2 * sy + 1])};
    const double rec = e_pme ? kc * e_pme[2 * sy] : 0.0;
    const double self = e_pme ? kc * e_pme[2 * sy + 1] : 0.0;
    const double eb = bonded ? Acc<T>::get(&bonded[3 * natoms]) : 0.0;
    const double ea = bonded ? Acc<T>::get(&bonded[3 * natoms + 1]) : 0.0;
    const double tot = e_tile[0] + e_tile[1] + rec + self + eb + ea;
    if (energy) energy[sy] = tot;
    if (terms) {
      const int nt = bonded ? 6 : 4;
      terms[nt * sy] = e_tile[0];
      terms[nt * sy + 1] = e_tile[1];
      terms[nt * sy + 2] = rec;
      terms[nt * sy + 3] = self;
      if (bonded) {
        terms[nt * sy + 4] = eb;
        terms[nt * sy + 5] = ea;
      }
    }
  }
}

template <class T>
__global__ void cast_inputs_kernel(const double *x64, const double *box64, T *x, T *box, int64_t n3) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n3; k += (int64_t)gridDim.x * blockDim.x)
    x[k] = (T)x64[k];
  if (blockIdx.x == 0 && threadIdx.x < 9) box[threadIdx.x] = (T)box64[threadIdx.x];
}

// Host-side B-spline moduli theta(k) = sum_{m=-3}^{2} M6(m+3) cos(2 pi m k / K)
// (torchff/bsplines.py:20-63), with M6 at the integers from the same recursion as the
// device splines.
// Launches the tile kernel of a mode; FP64 with the polynomial range that covers alpha rc.
template <class T, int MODE>
int launch_tile(bool pdl, int64_t max_items, int sms, cudaStream_t s, const TileArgs<T> &A) {
  constexpr int NW = TileCfg<T, MODE>::NW;
  const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((max_items + NW - 1) / NW, (int64_t)sms * 48 / NW));
  if constexpr (sizeof(T) == 8) {
    switch (erf_range(A.alpha, A.rc)) {
      case kErfShort: return launch_k(pdl, tile_kernel<T, MODE, kErfShort>, nb, NW * kWarp, 0, s, A);
      case kErfLong: return launch_k(pdl, tile_kernel<T, MODE, kErfLong>, nb, NW * kWarp, 0, s, A);
      default: break;
    }
  }
  return launch_k(pdl, tile_kernel<T, MODE, kErfLibrary>, nb, NW * kWarp, 0, s, A);
}

inline void host_bspline6_at_integers(double val[6]) {
  double m[6] = {0, 1, 0, 0, 0, 0};  // M2(0)=0, M2(1)=1
  for (int n = 3; n <= 6; ++n) {
    double nm[6] = {0};
    for (int k = 0; k < n; ++k) {
      const double cur = (k < n - 1) ? m[k] : 0.0;
      const double prev = (k > 0) ? m[k - 1] : 0.0;
      nm[k] = ((double)k * cur + (double)(n - k) * prev) / (double)(n - 1);
    }
    for (int k = 0; k < 6; ++k) m[k] = nm[k];
  }
  for (int k = 0; k < 6; ++k) val[k] = m[k];
}

inline std::vector<double> host_moduli(int K, int count) {
  double b[6];
  host_bspline6_at_integers(b);
  std::vector<double> out(count);
  for (int k = 0; k < count; ++k) {
    double s = 0.0;
    for (int m = -3; m < 3; ++m) s += b[m + 3] * std::cos(2.0 * M_PI * m * k / K);
    out[k] = s;
  }
  return out;
}

}  // namespace
}  // namespace tff

#include "pair_tile.cuh"
