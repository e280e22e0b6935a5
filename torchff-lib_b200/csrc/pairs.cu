// Pair terms over an explicit (P, 2) pair list: the drop-in kernels behind
// compute_nonbonded_energy_from_atom_pairs, compute_nonbonded_forces_from_atom_pairs,
// compute_coulomb_energy, compute_lennard_jones_energy and rank-0
// compute_multipolar_energy_from_atom_pairs.
//
// A call is three launches: pair_prep_kernel clears the accumulators and packs every atom's
// operands into one 16-byte (FP64: 32-byte) record where the workspace has room for them, pair_kernel
// evaluates one pair per lane, pair_finish_kernel converts the accumulators into the caller's arrays.
// The work partition - and with it every summation order - depends on the sizes alone.
// Energies: per-thread FP64, fixed-order block and grid reduction. Gradients: int64
// fixed-point atomics in mixed precision (order-independent, bit-reproducible), FP64
// atomics in FP64 mode.
#include <math.h>

#include <mutex>

#include <cuda.h>   // driver types only: cuCtxGetCurrent / cuCtxGetId are reached via the runtime

#include <algorithm>

#include "cluster.cuh"
#include "erf_poly.cuh"

namespace tff {
namespace {

enum CoulMode { C_NONE = 0, C_SHIFT = 1, C_PLAIN = 2, C_EWALD = 3 };
enum LjMode { L_NONE = 0, L_ATOM = 1, L_PAIR = 2, L_TYPE = 3 };

constexpr int kPairBlock = 256;

template <class T> struct LjRec;
template <> struct LjRec<float> { using type = float2; };
template <> struct LjRec<double> { using type = double2; };

// Box of a call in the pair arithmetic's precision.
template <class T>
struct PairBox {
  T m[9], inv[9];
  int ortho;  // every off-diagonal element is zero
};

template <class T>
struct PairArgs {
  const typename V4<T>::type *atoms;    // (x, y, z, charge); L_TYPE: the type index in the last word.
                                        // FP32 L_ATOM: two per atom, the second (sigma, epsilon, 0, 0).
                                        // NULL: no records, the caller's arrays below are read
  const typename LjRec<T>::type *lj;    // FP64 L_ATOM: (sigma, epsilon)
  const PairBox<T> *box;                // NULL: open boundaries
  const int64_t *pairs;
  int64_t npairs;
  const int64_t *excl;
  int64_t nexcl;
  const T *x, *q;
  const int64_t *types;
  const T *sig, *eps;                   // L_ATOM: per atom; L_PAIR: per pair; L_TYPE: tables
  int64_t ntypes;
  double k, rc, alpha;
  typename Acc<T>::S *acc;              // (natoms, 4): dE/dx, dE/dy, dE/dz, dE/dq; NULL: none of them
  bool want_x, want_q;
  typename Acc<T>::S *acc_lj;           // L_ATOM: (natoms, 2): dE/dsigma, dE/depsilon; NULL: neither
  bool want_s, want_e;
  typename Acc<T>::S *gs, *ge;          // L_TYPE: table accumulators (nullable)
  T *gs_pair, *ge_pair;                 // per-pair parameter gradients (L_PAIR)
  int iters;                            // consecutive rows per lane (at most kMaxPairIters)
  double *partials;
  unsigned *ticket;
  double *energy;
};

__device__ __forceinline__ float type_bits(float, int t) { return __int_as_float(t); }
__device__ __forceinline__ double type_bits(double, int t) { return (double)t; }
__device__ __forceinline__ int bits_type(float w) { return __float_as_int(w); }
__device__ __forceinline__ int bits_type(double w) { return (int)w; }

// Clears the accumulators and the reduction ticket, packs the records of n atoms (0: none) and the box.
template <class T>
__global__ void __launch_bounds__(kPairBlock) pair_prep_kernel(int64_t n, const T *x, const T *q, const int64_t *types,
                                                               const T *sig, const T *eps, const T *box,
                                                               typename V4<T>::type *atoms,
                                                               bool wide, typename LjRec<T>::type *lj,
                                                               PairBox<T> *box_out,
                                                               ulonglong2 *acc, int64_t nacc2, unsigned *ticket) {
  pdl_enter();
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  if (t0 == 0) {
    *ticket = 0u;
    if (box) {
      Box b;
      load_box(box, b);
      for (int k = 0; k < 9; ++k) {
        box_out->m[k] = (T)b.m[k];
        box_out->inv[k] = (T)b.inv[k];
      }
      const double *m = b.m;
      box_out->ortho = m[1] == 0.0 && m[2] == 0.0 && m[3] == 0.0 && m[5] == 0.0 && m[6] == 0.0 && m[7] == 0.0;
    }
  }
  for (int64_t k = t0; k < nacc2; k += stride) acc[k] = make_ulonglong2(0ull, 0ull);
  for (int64_t i = t0; i < n; i += stride) {
    const T w = q ? q[i] : (types ? type_bits(T(0), (int)types[i]) : T(0));
    const auto rec = make_v4(x[3 * i], x[3 * i + 1], x[3 * i + 2], w);
    if (wide) {
      atoms[2 * i] = rec;
      atoms[2 * i + 1] = make_v4(sig[i], eps[i], T(0), T(0));
      continue;
    }
    atoms[i] = rec;
    if (lj) {
      typename LjRec<T>::type r;
      r.x = sig[i];
      r.y = eps[i];
      lj[i] = r;
    }
  }
}

// Accumulated value of a contribution: int64 fixed point (FP32) or the value itself (FP64).
template <class T> struct Contrib;
template <> struct Contrib<float> {
  using S = unsigned long long;
  using S2 = ulonglong2;
  static __device__ __forceinline__ S of(float v) { return to_fix_f(v); }
  static __device__ __forceinline__ S minus(S v) { return 0ull - v; }
};
template <> struct Contrib<double> {
  using S = double;
  using S2 = double2;
  static __device__ __forceinline__ S of(double v) { return v; }
  static __device__ __forceinline__ S minus(S v) { return -v; }
};

constexpr unsigned kNoRow = 0xffffffffu;  // no accumulator row (rows are counted in 32 bits)

__device__ __forceinline__ float erfc_t(float x) { return erfcf(x); }
__device__ __forceinline__ double erfc_t(double x) { return erfc(x); }
__device__ __forceinline__ float exp_t(float x) { return expf(x); }
__device__ __forceinline__ double exp_t(double x) { return exp(x); }
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt(x); }
__device__ __forceinline__ float sqrt_t(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_t(double x) { return sqrt(x); }

// FP32 L_ATOM calls read an atom's six operands as one 32-byte record.
template <class T, int LM> constexpr bool kWideRec = sizeof(T) == 4 && LM == L_ATOM;

// Record of atom i; `lj` only for L_ATOM.
template <class T, int LM, bool RECORDS>
__device__ __forceinline__ void load_atom(const PairArgs<T> &a, unsigned i, typename V4<T>::type &r,
                                          typename LjRec<T>::type &lj) {
  if constexpr (!RECORDS) {
    const T w = a.q ? a.q[i] : (a.types ? type_bits(T(0), (int)a.types[i]) : T(0));
    r = make_v4(a.x[3 * (int64_t)i], a.x[3 * (int64_t)i + 1], a.x[3 * (int64_t)i + 2], w);
    if (LM == L_ATOM) {
      lj.x = a.sig[i];
      lj.y = a.eps[i];
    }
  } else if constexpr (kWideRec<T, LM>) {
    float u, v;
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w), "=f"(lj.x), "=f"(lj.y), "=f"(u), "=f"(v)
                 : "l"(a.atoms + 2 * (int64_t)i));
  } else {
    r = a.atoms[i];
    if (LM == L_ATOM) lj = a.lj[i];
  }
}

// Adds the NC values of each lane's row (ids: accumulator row or kNoRow) into rows of NC
// accumulators. 32 / NC rows go per instruction, their values on neighbouring lanes, so that the
// NC atomics of a row reach L2 as one 32-byte (16-byte) sector.
template <int NC, class S>
__device__ __forceinline__ void add_rows(S *acc, const unsigned *ids, const S *vals, bool on, int lane) {
  constexpr int kPer = kWarp / NC;
#pragma unroll
  for (int r = 0; r < NC; ++r) {
    const int e = r * kPer + lane / NC;
    const unsigned id = ids[e];
    if (on && id != kNoRow) atomicAdd(&acc[(int64_t)NC * id + lane % NC], vals[NC * e + lane % NC]);
  }
}

// Rows per lane: enough that the sums of a run of rows over one atom stay in registers, few
// enough that the warps of the grid get even shares.
constexpr int kMaxPairIters = 8;

// Staged rows of a warp: row r at r + r / 8, so that lanes reading rows 8 l + u hit distinct banks.
constexpr int kStagedRows = kWarp * kMaxPairIters + kWarp * kMaxPairIters / 8;

// A warp stages 32 x `iters` consecutive rows; lane l evaluates rows l iters .. (l + 1) iters - 1
// one after another. Neighbour lists are written in runs of rows over one atom: the lane keeps
// the sums of that atom (the key) in registers while consecutive rows hold it, in either column,
// and adds them when it changes. The other end's values pass through shared memory so that the
// three (four with dE/dq) values of an atom sit on neighbouring lanes: one L2 sector per row
// and end instead of one per value. Rows whose force and charge gradients are zero (LJ of a type
// with epsilon 0) add nothing. In fixed point the sums are the same integers in any order.
// One atomic per value, eight memory clears and conversions per call before: a call over 20.8 M
// rows (99,000 atoms, FP32) 1,015 -> 515 us, 1.9 M rows of LJ and Ewald (9,000 atoms) 115 and
// 122 -> 42 and 60 us.
// ERF (FP64 Ewald): how erfc is evaluated (erf_poly.cuh). RECORDS: operands from the packed records.
template <class T, int CM, int LM, int ERF, bool RECORDS>
__global__ void __launch_bounds__(kPairBlock, sizeof(T) == 4 ? 4 : 3) pair_kernel(PairArgs<T> a) {
  pdl_enter();
  using A = Acc<T>;
  using C = Contrib<T>;
  using S = typename C::S;
  constexpr int W = kPairBlock / kWarp;
  constexpr bool kLj = LM == L_ATOM;
  __shared__ PairBox<T> s_box;
  __shared__ uint2 s_rows[W][kStagedRows];
  __shared__ __align__(16) S s_val[W][kWarp * 4];
  __shared__ unsigned s_id[W][kWarp];
  const bool periodic = a.box != nullptr;
  if (threadIdx.x < 9 && periodic) {
    s_box.m[threadIdx.x] = a.box->m[threadIdx.x];
    s_box.inv[threadIdx.x] = a.box->inv[threadIdx.x];
    if (threadIdx.x == 0) s_box.ortho = a.box->ortho;
  }
  __syncthreads();
  const bool ortho = periodic && s_box.ortho;
  const T bx = s_box.m[0], by = s_box.m[4], bz = s_box.m[8], ix = s_box.inv[0], iy = s_box.inv[4], iz = s_box.inv[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  S *val = s_val[w];
  unsigned *ids = s_id[w];
  uint2 *rows = s_rows[w];

  const T rc = (T)a.rc;
  const T rc2 = rc * rc;
  const T kc = (T)a.k;
  const T inv_rc = T(1) / rc;
  const T alpha = (T)a.alpha;
  const T two_a_rpi = (T)(2.0 * a.alpha / 1.7724538509055160273);
  const EwaldPoly<ERF == kErfLibrary ? kErfShort : ERF> ewald(a.alpha);  // unused with kErfLibrary
  double e_acc = 0.0;
  const bool grads = a.acc != nullptr, lj_grads = kLj && a.acc_lj != nullptr;

  const int64_t total = a.npairs + ((CM == C_EWALD) ? a.nexcl : 0);
  const int64_t nwarps = (int64_t)gridDim.x * W, per = (int64_t)a.iters * kWarp;
  for (int64_t base = ((int64_t)blockIdx.x * W + w) * per; base < total; base += nwarps * per) {
    __syncwarp();
    for (int u = 0; u < a.iters; ++u) {
      const int r = u * kWarp + lane;
      const int64_t t = base + r;
      uint2 row = make_uint2(kNoRow, kNoRow);
      if (t < total) {
        const bool ex = (CM == C_EWALD) && t >= a.npairs;
        const int64_t p = ex ? t - a.npairs : t;
        const int64_t *pl = ex ? a.excl : a.pairs;
        const int64_t i = pl[2 * p], j = pl[2 * p + 1];
        if (i >= 0 && j >= 0) row = make_uint2((unsigned)i, (unsigned)j);
      }
      rows[r + (r >> 3)] = row;
    }
    __syncwarp();
    unsigned key = kNoRow;            // atom whose sums the lane holds
    S ks[4] = {}, kp[2] = {};         // its dE/dx, dE/dq; dE/dsigma, dE/depsilon
    const auto flush = [&]() {
      if (key == kNoRow) return;
      if (grads) {
        if (a.want_x) {
#pragma unroll
          for (int c = 0; c < 3; ++c) atomicAdd(&a.acc[4 * (int64_t)key + c], ks[c]);
        }
        if (CM != C_NONE && a.want_q) atomicAdd(&a.acc[4 * (int64_t)key + 3], ks[3]);
#pragma unroll
        for (int c = 0; c < 4; ++c) ks[c] = S(0);
      }
      if (lj_grads) {
        if (a.want_s) atomicAdd(&a.acc_lj[2 * (int64_t)key], kp[0]);
        if (a.want_e) atomicAdd(&a.acc_lj[2 * (int64_t)key + 1], kp[1]);
        kp[0] = kp[1] = S(0);
      }
    };
#pragma unroll 1
    for (int u = 0; u < a.iters; ++u) {
      const int r = lane * a.iters + u;
      const uint2 row = rows[r + (r >> 3)];
      const unsigned i = row.x, j = row.y;
      const int64_t t = base + r;
      const bool is_excl = (CM == C_EWALD) && (t >= a.npairs);
      bool in = i != kNoRow;
      T fx = T(0), fy = T(0), fz = T(0), gqi = T(0), gqj = T(0), gsv = T(0), gei = T(0), gej = T(0);
      if (in) {
        typename V4<T>::type pi, pj;
        typename LjRec<T>::type li{}, lj{};
        load_atom<T, LM, RECORDS>(a, i, pi, li);
        load_atom<T, LM, RECORDS>(a, j, pj, lj);
        T dx = pi.x - pj.x;
        T dy = pi.y - pj.y;
        T dz = pi.z - pj.z;
        if (ortho) {  // min_image without the products by zero
          T sa = dx * ix, sb = dy * iy, sc = dz * iz;
          sa -= floor(sa + T(0.5));
          sb -= floor(sb + T(0.5));
          sc -= floor(sc + T(0.5));
          dx = sa * bx;
          dy = sb * by;
          dz = sc * bz;
        } else if (periodic) {
          min_image(dx, dy, dz, s_box.m, s_box.inv);
        }
        const T r2 = dx * dx + dy * dy + dz * dz;
        in = r2 <= rc2;
        if (in) {
          const T rinv = rsqrt_t(r2);
          const T rinv2 = rinv * rinv;
          T e = T(0);
          T dedr_over_r = T(0);  // (dE/dr) / r

          if (CM != C_NONE) {
            const T qi = pi.w, qj = pj.w;
            T f;       // energy per unit k q_i q_j
            T dfdr_r;  // (df/dr) / r
            if (CM == C_SHIFT) {
              f = rinv - inv_rc;
              dfdr_r = -rinv2 * rinv;
            } else if (CM == C_PLAIN) {
              f = rinv;
              dfdr_r = -rinv2 * rinv;
            } else if constexpr (ERF != kErfLibrary) {
              T g, tx;
              if (is_excl)
                ewald.excluded(r2, f, g);
              else
                ewald.eval(r2, rinv, rinv2, f, g, tx);
              dfdr_r = -g;
            } else {
              const T r = r2 * rinv;
              const T u = alpha * r;
              T damp = erfc_t(u);
              if (is_excl) damp -= T(1);
              f = damp * rinv;
              dfdr_r = -(damp * rinv2 + two_a_rpi * exp_t(-u * u) * rinv) * rinv;
            }
            e += kc * qi * qj * f;
            dedr_over_r += kc * qi * qj * dfdr_r;
            gqi = kc * qj * f;
            gqj = kc * qi * f;
          }

          if (LM != L_NONE && !is_excl) {
            T s, ep, sqe_i = T(0), sqe_j = T(0);
            int64_t tidx = 0;
            if (LM == L_ATOM) {
              s = T(0.5) * (li.x + lj.x);
              sqe_i = li.y;
              sqe_j = lj.y;
              ep = sqrt_t(sqe_i * sqe_j);
            } else if (LM == L_PAIR) {
              s = a.sig[t];
              ep = a.eps[t];
            } else {
              tidx = bits_type(pi.w) * a.ntypes + bits_type(pj.w);
              s = a.sig[tidx];
              ep = a.eps[tidx];
            }
            const T sr2 = s * s * rinv2;
            const T sr6 = sr2 * sr2 * sr2;
            e += T(4) * ep * sr6 * (sr6 - T(1));
            const T g = T(24) * ep * sr6 * (T(2) * sr6 - T(1));  // = -r dE/dr = s dE/ds
            dedr_over_r -= g * rinv2;
            if (LM == L_ATOM) {
              if (lj_grads) {
                gsv = T(0.5) * (g / s);
                if (ep > T(0)) {
                  const T h = T(4) * sr6 * (sr6 - T(1)) / (T(2) * ep);
                  gei = h * sqe_j;
                  gej = h * sqe_i;
                }
              }
            } else if (LM == L_PAIR) {
              if (a.gs_pair) a.gs_pair[t] = g / s;
              if (a.ge_pair) a.ge_pair[t] = T(4) * sr6 * (sr6 - T(1));
            } else {
              if (a.gs) A::add(&a.gs[tidx], (double)(g / s));
              if (a.ge) A::add(&a.ge[tidx], (double)(T(4) * sr6 * (sr6 - T(1))));
            }
          }
          e_acc += (double)e;
          fx = dedr_over_r * dx;
          fy = dedr_over_r * dy;
          fz = dedr_over_r * dz;
        }
      }
      if (LM == L_PAIR && !in && t < a.npairs) {
        if (a.gs_pair) a.gs_pair[t] = T(0);
        if (a.ge_pair) a.ge_pair[t] = T(0);
      }
      if (!grads && !lj_grads) continue;
      const bool some = in && (lj_grads || fx != T(0) || fy != T(0) || fz != T(0) || gqi != T(0) || gqj != T(0));
      unsigned other = kNoRow;
      bool swap = false;  // the key is j
      if (some) {
        if (key != i && key != j) {
          flush();
          // the new key: the end that the lane's next row holds too
          const int rn = min(r + 1, lane * a.iters + a.iters - 1);
          const uint2 next = rows[rn + (rn >> 3)];
          key = u + 1 < a.iters && (next.x == j || next.y == j) && next.x != i && next.y != i ? j : i;
        }
        swap = key != i;
        other = swap ? i : j;
      }
      if (!__any_sync(kFull, some)) continue;
      if (grads) {
        // dE/dx of i is +f, of j -f
        const S vx = C::of(fx), vy = C::of(fy), vz = C::of(fz);
        const S mx = C::minus(vx), my = C::minus(vy), mz = C::minus(vz);
        ks[0] += swap ? mx : vx;
        ks[1] += swap ? my : vy;
        ks[2] += swap ? mz : vz;
        S vq = S(0);
        if (CM != C_NONE) {
          ks[3] += C::of(swap ? gqj : gqi);
          vq = C::of(swap ? gqi : gqj);
        }
        using S2 = typename C::S2;
        reinterpret_cast<S2 *>(val)[2 * lane] = S2{swap ? vx : mx, swap ? vy : my};
        reinterpret_cast<S2 *>(val)[2 * lane + 1] = S2{swap ? vz : mz, vq};
        ids[lane] = other;
        __syncwarp();
        add_rows<4>(a.acc, ids, val, (lane & 3) == 3 ? CM != C_NONE && a.want_q : a.want_x, lane);
        __syncwarp();
      }
      if (lj_grads) {
        const S vs = C::of(gsv);
        kp[0] += vs;
        kp[1] += C::of(swap ? gej : gei);
        val[2 * lane] = vs;
        val[2 * lane + 1] = C::of(swap ? gei : gej);
        ids[lane] = other;
        __syncwarp();
        add_rows<2>(a.acc_lj, ids, val, (lane & 1) ? a.want_e : a.want_s, lane);
        __syncwarp();
      }
    }
    flush();
  }
  grid_sum<kPairBlock>(e_acc, a.partials, a.ticket, a.energy, false);
}

// Accumulators -> the caller's arrays: gx[k] = gx_scale * acc (or += with gx_add), the others as
// they are; the energy scalar.
template <class T>
struct PairOut {
  const typename Acc<T>::S *acc, *acc_lj, *gs_tab, *ge_tab;
  T *gx, *gq, *gs, *ge;  // nullable
  double gx_scale;
  bool gx_add;
  int64_t natoms, ntab;
  const double *e;
  T *energy;  // nullable
  double e_scale;
};

template <class T>
__global__ void __launch_bounds__(kPairBlock) pair_finish_kernel(PairOut<T> a) {
  pdl_enter();
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  if (a.gx)
    for (int64_t k = t0; k < 3 * a.natoms; k += stride) {
      const int64_t i = k / 3;
      const double v = a.gx_scale * Acc<T>::get(&a.acc[4 * i + (k - 3 * i)]);
      a.gx[k] = a.gx_add ? (T)((double)a.gx[k] + v) : (T)v;
    }
  if (a.gq)
    for (int64_t i = t0; i < a.natoms; i += stride) a.gq[i] = (T)Acc<T>::get(&a.acc[4 * i + 3]);
  if (a.acc_lj)
    for (int64_t i = t0; i < a.natoms; i += stride) {
      if (a.gs) a.gs[i] = (T)Acc<T>::get(&a.acc_lj[2 * i]);
      if (a.ge) a.ge[i] = (T)Acc<T>::get(&a.acc_lj[2 * i + 1]);
    }
  for (int64_t i = t0; i < a.ntab; i += stride) {
    if (a.gs) a.gs[i] = (T)Acc<T>::get(&a.gs_tab[i]);
    if (a.ge) a.ge[i] = (T)Acc<T>::get(&a.ge_tab[i]);
  }
  if (t0 == 0 && a.energy) a.energy[0] = (T)(a.e_scale * a.e[0]);
}

// The records of a workspace are read as 16- and 32-byte vectors: its parts are laid out from the
// first multiple of this in it.
constexpr size_t kWsAlign = 256;

struct PairLayout {
  size_t acc, acc_lj, gs_tab, ge_tab, acc_end;  // accumulators, from offset 0
  size_t atoms, lj, box, partials, ticket, energy, bytes;
};

// Accumulators: 4 per atom (dE/dx, dE/dq), then 2 per atom (dE/dsigma, dE/depsilon) or the type
// tables'; both accumulator types are 8 bytes. Without records the layout takes the 48 bytes per atom
// (6 accumulators) and 64.5 KiB that callers of earlier versions of the library reserve: a smaller
// workspace than tff_pairs_workspace_bytes names is then still enough, and the kernel reads the caller's
// arrays (the same results; 20.9 M rows over 99,000 atoms with all gradients, FP32: 732 us, with records 687).
PairLayout pair_layout(int dtype, int64_t natoms, int64_t ntypes, bool records) {
  const size_t ts = dtype == TFF_F64 ? 8 : 4, tab = (size_t)(ntypes * ntypes) * 8;
  PairLayout L{};
  Carver c(nullptr);
  const auto take = [&c](size_t bytes) {
    c.take<char>(bytes);
    return c.off - bytes;
  };
  if (!records) {
    const size_t atom = (size_t)natoms * 8;
    L.acc_lj = L.gs_tab = 4 * atom;
    L.ge_tab = L.gs_tab + tab;
    L.acc_end = 4 * atom + 2 * std::max(atom, tab);
    take(L.acc_end);
    L.bytes = c.bytes() + 8192 * sizeof(double) + 512;
    L.box = take(18 * ts + 8);
    L.ticket = take(sizeof(unsigned));
    L.energy = take(sizeof(double));
    L.partials = take(8064 * sizeof(double));  // with room to align the caller's pointer
    return L;
  }
  L.acc = take((size_t)natoms * 4 * 8);
  L.acc_lj = take((size_t)natoms * 2 * 8);
  L.gs_tab = take(tab);
  L.ge_tab = take(tab);
  L.atoms = L.acc_end = take((size_t)natoms * 32);  // FP64 (x, y, z, q), or FP32 with room for a second vector
  L.lj = take(dtype == TFF_F64 ? (size_t)natoms * 16 : 0);
  L.box = take(18 * ts + 8);
  L.partials = take(8 * 1024 * sizeof(double));
  L.ticket = take(sizeof(unsigned));
  L.energy = take(sizeof(double));
  L.bytes = c.bytes() + kWsAlign;  // room to align the caller's pointer
  return L;
}

int grid_blocks(int64_t work) {
  int64_t want = (work + kPairBlock - 1) / kPairBlock;
  int64_t cap = (int64_t)sm_count() * 8;
  if (want < 1) want = 1;
  return (int)std::min(want, cap);
}

template <class T, int CM, int LM, int ERF = kErfLibrary>
int launch_pairs(PairArgs<T> a, int64_t total, cudaStream_t s) {
  const int nb = grid_blocks(total);
  const int64_t share = (total + (int64_t)nb * kPairBlock - 1) / ((int64_t)nb * kPairBlock);
  a.iters = (int)std::max<int64_t>(1, std::min<int64_t>(kMaxPairIters, share));
  const auto kernel = a.atoms ? pair_kernel<T, CM, LM, ERF, true> : pair_kernel<T, CM, LM, ERF, false>;
  return launch_k(true, kernel, nb, kPairBlock, 0, s, a);
}

template <class T>
int dispatch_pairs(int cm, int lm, const PairArgs<T> &a, int64_t total, cudaStream_t s) {
#define TFF_PAIR_CASE(C, L) \
  if (cm == C && lm == L) return launch_pairs<T, C, L>(a, total, s);
  TFF_PAIR_CASE(C_SHIFT, L_ATOM)
  TFF_PAIR_CASE(C_PLAIN, L_ATOM)
  TFF_PAIR_CASE(C_SHIFT, L_NONE)
  TFF_PAIR_CASE(C_PLAIN, L_NONE)
  if constexpr (sizeof(T) == 8)
    if (cm == C_EWALD && lm == L_NONE) {
      const ErfRange range = erf_range(a.alpha, a.rc);
      if (range == kErfShort) return launch_pairs<T, C_EWALD, L_NONE, kErfShort>(a, total, s);
      if (range == kErfLong) return launch_pairs<T, C_EWALD, L_NONE, kErfLong>(a, total, s);
    }
  TFF_PAIR_CASE(C_EWALD, L_NONE)
  TFF_PAIR_CASE(C_NONE, L_PAIR)
  TFF_PAIR_CASE(C_NONE, L_TYPE)
#undef TFF_PAIR_CASE
  set_error("unsupported pair-term combination");
  return TFF_ERR_INVALID;
}

// Common driver: zero accumulators, run the pair kernel, convert outputs.
struct PairCall {
  int dtype;
  int cm, lm;
  int64_t natoms, npairs, nexcl, ntypes;
  const void *x, *box, *q, *sig, *eps;
  const int64_t *pairs, *excl, *types;
  double k, rc, alpha;
  void *energy;       // T scalar (nullable)
  double e_scale;
  void *gx; double gx_scale; bool gx_add;
  void *gq, *gs, *ge; // T outputs (per atom / per table / per pair)
  void *ws; size_t ws_bytes;
};

template <class T>
int run_pairs(const PairCall &c, cudaStream_t s) {
  using S = typename Acc<T>::S;
  PairLayout L = pair_layout(c.dtype, c.natoms, c.ntypes, true);
  const bool records = c.ws_bytes >= L.bytes;
  if (!records) L = pair_layout(c.dtype, c.natoms, c.ntypes, false);
  if (c.ws_bytes < L.bytes || c.ws == nullptr) {
    set_error("workspace too small: need %zu bytes, got %zu", L.bytes, c.ws_bytes);
    return TFF_ERR_WORKSPACE;
  }
  char *ws = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(c.ws) + kWsAlign - 1) & ~uintptr_t(kWsAlign - 1));
  PairArgs<T> a{};
  auto *atoms = records ? reinterpret_cast<typename V4<T>::type *>(ws + L.atoms) : nullptr;
  const bool wide = sizeof(T) == 4 && c.lm == L_ATOM;
  auto *lj = records && c.lm == L_ATOM && !wide ? reinterpret_cast<typename LjRec<T>::type *>(ws + L.lj) : nullptr;
  auto *box = reinterpret_cast<PairBox<T> *>(ws + L.box);
  a.atoms = atoms;
  a.lj = lj;
  a.box = c.box ? box : nullptr;
  a.pairs = c.pairs;
  a.npairs = c.npairs;
  a.excl = c.excl;
  a.nexcl = c.nexcl;
  a.x = static_cast<const T *>(c.x);
  a.q = c.cm != C_NONE ? static_cast<const T *>(c.q) : nullptr;
  a.types = c.lm == L_TYPE ? c.types : nullptr;
  a.sig = static_cast<const T *>(c.sig);
  a.eps = static_cast<const T *>(c.eps);
  a.ntypes = c.ntypes;
  a.k = c.k;
  a.rc = c.rc;
  a.alpha = c.alpha;
  a.want_x = c.gx != nullptr;
  a.want_q = c.gq != nullptr;
  a.acc = c.gx || c.gq ? reinterpret_cast<S *>(ws + L.acc) : nullptr;
  a.want_s = c.gs != nullptr;
  a.want_e = c.ge != nullptr;
  if (c.lm == L_ATOM && (c.gs || c.ge)) a.acc_lj = reinterpret_cast<S *>(ws + L.acc_lj);
  if (c.lm == L_TYPE) {
    a.gs = c.gs ? reinterpret_cast<S *>(ws + L.gs_tab) : nullptr;
    a.ge = c.ge ? reinterpret_cast<S *>(ws + L.ge_tab) : nullptr;
  }
  if (c.lm == L_PAIR) {
    a.gs_pair = static_cast<T *>(c.gs);
    a.ge_pair = static_cast<T *>(c.ge);
  }
  a.partials = reinterpret_cast<double *>(ws + L.partials);
  a.ticket = reinterpret_cast<unsigned *>(ws + L.ticket);
  a.energy = reinterpret_cast<double *>(ws + L.energy);
  // the accumulator region is cleared as far as this call uses it
  const size_t zero = a.acc_lj || a.gs || a.ge ? L.acc_end : a.acc ? L.acc_lj : 0;
  const int64_t nacc2 = (int64_t)(zero / sizeof(ulonglong2));
  const auto blocks = [](int64_t work) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((work + kPairBlock - 1) / kPairBlock, (int64_t)sm_count() * 8));
  };
  int st = launch_k(false, pair_prep_kernel<T>, blocks(std::max(c.natoms, nacc2)), kPairBlock, 0, s,
                    records ? c.natoms : (int64_t)0, a.x, a.q, a.types, a.sig, a.eps, static_cast<const T *>(c.box),
                    atoms, wide, lj, box, reinterpret_cast<ulonglong2 *>(ws), nacc2, a.ticket);
  if (st != TFF_OK) return st;
  const int64_t total = c.npairs + (c.cm == C_EWALD ? c.nexcl : 0);
  if ((st = dispatch_pairs<T>(c.cm, c.lm, a, total, s)) != TFF_OK) return st;
  PairOut<T> o{};
  o.acc = a.acc;
  o.acc_lj = a.acc_lj;
  o.gs_tab = a.gs;
  o.ge_tab = a.ge;
  o.gx = static_cast<T *>(c.gx);
  o.gq = static_cast<T *>(c.gq);
  o.gs = c.lm == L_PAIR ? nullptr : static_cast<T *>(c.gs);
  o.ge = c.lm == L_PAIR ? nullptr : static_cast<T *>(c.ge);
  o.gx_scale = c.gx_scale;
  o.gx_add = c.gx_add;
  o.natoms = c.natoms;
  o.ntab = c.lm == L_TYPE && (c.gs || c.ge) ? c.ntypes * c.ntypes : 0;
  o.e = a.energy;
  o.energy = static_cast<T *>(c.energy);
  o.e_scale = c.e_scale;
  const int64_t work = o.gx ? 3 * c.natoms : o.gq || o.acc_lj ? c.natoms : 1;
  return launch_k(true, pair_finish_kernel<T>, blocks(std::max(work, o.ntab)), kPairBlock, 0, s, o);
}

int run_pairs_any(const PairCall &c, cudaStream_t s) {
  TFF_ARG(c.dtype == TFF_F32 || c.dtype == TFF_F64, "dtype must be TFF_F32 or TFF_F64");
  TFF_ARG(c.natoms >= 0 && c.npairs >= 0 && c.nexcl >= 0, "negative sizes");
  TFF_ARG(c.x != nullptr || c.natoms == 0, "coords is NULL");
  TFF_ARG(c.pairs != nullptr || c.npairs == 0, "pairs is NULL");
  TFF_ARG(c.rc > 0.0, "cutoff must be positive");
  if (c.cm != C_NONE) TFF_ARG(c.q != nullptr, "charges is NULL");
  if (c.lm != L_NONE) TFF_ARG(c.sig != nullptr && c.eps != nullptr, "sigma/epsilon is NULL");
  if (c.lm == L_TYPE) TFF_ARG(c.types != nullptr && c.ntypes > 0, "atom_types/ntypes invalid");
  return c.dtype == TFF_F32 ? run_pairs<float>(c, s) : run_pairs<double>(c, s);
}

// ---------------------------------------------------------------------------------------
// Scratch for tff_nonbonded_atom_pairs_noalloc: a file-scope device array, so that caller
// never has to allocate. Sized for TFF_NOALLOC_MAX_ATOMS atoms (6 accumulators and 6 packed
// operands of 8 bytes per atom, the block partials, the box and the reduction ticket/energy,
// 6.1 MiB); every GPU that loads the library holds it until the process exits.
// ---------------------------------------------------------------------------------------
constexpr int64_t kNoAllocMaxAtoms = TFF_NOALLOC_MAX_ATOMS;
constexpr size_t kNoAllocScratchBytes = (size_t)kNoAllocMaxAtoms * 12 * 8 + 8192 * 8 + 12 * 256;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Id of the context current on this thread (0 while none is), through the driver's
// cuCtxGetCurrent / cuCtxGetId reached via the runtime (the library does not link the driver
// library). Context ids are unique for the life of the process, so the context the runtime
// creates after a cudaDeviceReset never carries the id of the one it replaced.
int current_context_id(unsigned long long *id) {
  using GetCurrent = CUresult (*)(CUcontext *);
  using GetId = CUresult (*)(CUcontext, unsigned long long *);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  if (get_current == nullptr || get_id == nullptr) {
    void *f1 = nullptr, *f2 = nullptr;
    cudaDriverEntryPointQueryResult r1 = cudaDriverEntryPointSymbolNotFound, r2 = r1;
    TFF_CUDA(cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &r1));
    TFF_CUDA(cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &r2));
    TFF_ARG(r1 == cudaDriverEntryPointSuccess && r2 == cudaDriverEntryPointSuccess && f1 && f2,
            "the driver offers no cuCtxGetCurrent/cuCtxGetId");
    get_current = reinterpret_cast<GetCurrent>(f1);
    get_id = reinterpret_cast<GetId>(f2);
  }
  CUcontext ctx = nullptr;
  TFF_ARG(get_current(&ctx) == CUDA_SUCCESS, "cuCtxGetCurrent failed");
  *id = 0;
  if (ctx != nullptr) TFF_ARG(get_id(ctx, id) == CUDA_SUCCESS, "cuCtxGetId failed");
  return TFF_OK;
}

// Device address of g_noalloc_scratch in the current device's context. In host code the
// symbol is only a host-side stand-in, so the address is looked up with
// cudaGetSymbolAddress (with that device current) at the first call on each device, and
// again whenever the device's context has changed since (after a cudaDeviceReset, the
// old address belongs to a destroyed context).
int noalloc_scratch(void **out) {
  static std::mutex mu;
  static void *addr[64] = {nullptr};
  static unsigned long long ctx_of[64] = {0};
  int dev = 0;
  TFF_CUDA(cudaGetDevice(&dev));
  TFF_ARG(dev >= 0 && dev < 64, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  unsigned long long ctx = 0;
  int st = current_context_id(&ctx);
  if (st != TFF_OK) return st;
  if (addr[dev] == nullptr || ctx == 0 || ctx != ctx_of[dev]) {
    void *p = nullptr;
    TFF_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));   // makes the context current if none was
    st = current_context_id(&ctx);
    if (st != TFF_OK) return st;
    addr[dev] = p;
    ctx_of[dev] = ctx;
  }
  *out = addr[dev];
  return TFF_OK;
}

}  // namespace
}  // namespace tff

using namespace tff;

extern "C" {

// Same computation as tff_nonbonded_atom_pairs, for callers that cannot allocate device
// memory: a force plugin inside a molecular-dynamics engine that owns every device
// allocation and hands the plugin only its input and output buffers, or a time-critical
// loop that must never reach an allocator (an allocation can synchronise the device or
// fail mid-run). Scratch is the library's static device array instead of a caller
// workspace; the caller still passes inputs and outputs. Limits and sharing:
// natoms <= TFF_NOALLOC_MAX_ATOMS (larger sizes return TFF_ERR_INVALID); the first call on
// each device (and the first after a device reset) looks the array up with
// cudaGetSymbolAddress, so make that first call before any stream capture; all calls share
// the one array (its accumulators are cleared at the start of every call and it keeps the
// last call's contents), so calls that overlap on the GPU, e.g. on two streams at once,
// race and must be serialised by the caller.
int tff_nonbonded_atom_pairs_noalloc(int dtype, int64_t natoms, const void *coords, int64_t npairs,
                                     const int64_t *pairs, const void *box, const void *sigma,
                                     const void *epsilon, const void *charges, double coul_constant,
                                     double cutoff, int do_shift, void *energy, void *grad_coords,
                                     void *grad_sigma, void *grad_epsilon, void *grad_charges,
                                     tff_stream_t stream) {
  TFF_ARG(natoms >= 0 && natoms <= kNoAllocMaxAtoms,
          "natoms=%lld exceeds the static scratch limit of %lld atoms of tff_nonbonded_atom_pairs_noalloc",
          (long long)natoms, (long long)kNoAllocMaxAtoms);
  const size_t need = pair_layout(dtype, natoms, 0, true).bytes;
  TFF_ARG(need <= kNoAllocScratchBytes, "static scratch too small (%zu > %zu bytes)", need, kNoAllocScratchBytes);
  void *ws = nullptr;
  int st = noalloc_scratch(&ws);
  if (st != TFF_OK) return st;
  PairCall c{};
  c.dtype = dtype;
  c.cm = do_shift ? C_SHIFT : C_PLAIN;
  c.lm = L_ATOM;
  c.natoms = natoms; c.npairs = npairs; c.x = coords; c.box = box; c.q = charges;
  c.sig = sigma; c.eps = epsilon; c.pairs = pairs; c.k = coul_constant; c.rc = cutoff;
  c.energy = energy; c.e_scale = 1.0;
  c.gx = grad_coords; c.gx_scale = 1.0; c.gx_add = false;
  c.gq = grad_charges; c.gs = grad_sigma; c.ge = grad_epsilon;
  c.ws = ws; c.ws_bytes = kNoAllocScratchBytes;
  return run_pairs_any(c, (cudaStream_t)stream);
}

size_t tff_pairs_workspace_bytes(int dtype, int64_t natoms, int64_t ntypes) {
  return pair_layout(dtype, natoms, ntypes, true).bytes;
}

int tff_nonbonded_atom_pairs(int dtype, int64_t natoms, const void *coords, int64_t npairs,
                             const int64_t *pairs, const void *box, const void *sigma,
                             const void *epsilon, const void *charges, double coul_constant,
                             double cutoff, int do_shift, void *energy, void *grad_coords,
                             void *grad_sigma, void *grad_epsilon, void *grad_charges,
                             void *workspace, size_t workspace_bytes, tff_stream_t stream) {
  TFF_NVTX("tff_nonbonded_atom_pairs");
  PairCall c{};
  c.dtype = dtype;
  c.cm = do_shift ? C_SHIFT : C_PLAIN;
  c.lm = L_ATOM;
  c.natoms = natoms; c.npairs = npairs; c.x = coords; c.box = box; c.q = charges;
  c.sig = sigma; c.eps = epsilon; c.pairs = pairs; c.k = coul_constant; c.rc = cutoff;
  c.energy = energy; c.e_scale = 1.0;
  c.gx = grad_coords; c.gx_scale = 1.0; c.gx_add = false;
  c.gq = grad_charges; c.gs = grad_sigma; c.ge = grad_epsilon;
  c.ws = workspace; c.ws_bytes = workspace_bytes;
  return run_pairs_any(c, (cudaStream_t)stream);
}

int tff_nonbonded_forces_atom_pairs(int dtype, int64_t natoms, const void *coords,
                                    int64_t npairs, const int64_t *pairs, const void *box,
                                    const void *sigma, const void *epsilon, const void *charges,
                                    double coul_constant, double cutoff, void *forces,
                                    void *workspace, size_t workspace_bytes, tff_stream_t stream) {
  TFF_NVTX("tff_nonbonded_forces_atom_pairs");
  TFF_ARG(forces != nullptr || natoms == 0, "forces is NULL");
  PairCall c{};
  c.dtype = dtype;
  c.cm = C_SHIFT;
  c.lm = L_ATOM;
  c.natoms = natoms; c.npairs = npairs; c.x = coords; c.box = box; c.q = charges;
  c.sig = sigma; c.eps = epsilon; c.pairs = pairs; c.k = coul_constant; c.rc = cutoff;
  c.gx = forces; c.gx_scale = -1.0; c.gx_add = true;
  c.ws = workspace; c.ws_bytes = workspace_bytes;
  return run_pairs_any(c, (cudaStream_t)stream);
}

int tff_coulomb_atom_pairs(int dtype, int64_t natoms, const void *coords, int64_t npairs,
                           const int64_t *pairs, const void *box, const void *charges,
                           double coul_constant, double cutoff, int do_shift, void *energy,
                           void *grad_coords, void *grad_charges, void *workspace,
                           size_t workspace_bytes, tff_stream_t stream) {
  TFF_NVTX("tff_coulomb_atom_pairs");
  PairCall c{};
  c.dtype = dtype;
  c.cm = do_shift ? C_SHIFT : C_PLAIN;
  c.lm = L_NONE;
  c.natoms = natoms; c.npairs = npairs; c.x = coords; c.box = box; c.q = charges;
  c.pairs = pairs; c.k = coul_constant; c.rc = cutoff;
  c.energy = energy; c.e_scale = 1.0;
  c.gx = grad_coords; c.gx_scale = 1.0;
  c.gq = grad_charges;
  c.ws = workspace; c.ws_bytes = workspace_bytes;
  return run_pairs_any(c, (cudaStream_t)stream);
}

int tff_lennard_jones_atom_pairs(int dtype, int64_t natoms, const void *coords, int64_t npairs,
                                 const int64_t *pairs, const void *box, const void *sigma,
                                 const void *epsilon, double cutoff, const int64_t *atom_types,
                                 int64_t ntypes, void *energy, void *grad_coords,
                                 void *grad_sigma, void *grad_epsilon, void *workspace,
                                 size_t workspace_bytes, tff_stream_t stream) {
  TFF_NVTX("tff_lennard_jones_atom_pairs");
  PairCall c{};
  c.dtype = dtype;
  c.cm = C_NONE;
  c.lm = atom_types ? L_TYPE : L_PAIR;
  c.natoms = natoms; c.npairs = npairs; c.x = coords; c.box = box;
  c.sig = sigma; c.eps = epsilon; c.types = atom_types; c.ntypes = atom_types ? ntypes : 0;
  c.pairs = pairs; c.rc = cutoff;
  c.energy = energy; c.e_scale = 1.0;
  c.gx = grad_coords; c.gx_scale = 1.0;
  c.gs = grad_sigma; c.ge = grad_epsilon;
  c.ws = workspace; c.ws_bytes = workspace_bytes;
  return run_pairs_any(c, (cudaStream_t)stream);
}

int tff_ewald_real_atom_pairs(int dtype, int64_t natoms, const void *coords, const void *box,
                              int64_t npairs, const int64_t *pairs, int64_t npairs_excl,
                              const int64_t *pairs_excl, const void *charges, double cutoff,
                              double ewald_alpha, double prefactor, void *energy,
                              void *grad_coords, void *grad_charges, void *workspace,
                              size_t workspace_bytes, tff_stream_t stream) {
  TFF_NVTX("tff_ewald_real_atom_pairs");
  PairCall c{};
  c.dtype = dtype;
  const bool ewald = ewald_alpha >= 0.0;
  c.cm = ewald ? C_EWALD : C_PLAIN;
  c.lm = L_NONE;
  c.natoms = natoms; c.npairs = npairs; c.x = coords; c.box = box; c.q = charges;
  c.pairs = pairs;
  // the exclusion correction only exists for a positive Ewald alpha (torchff/multipoles.py:317)
  c.excl = (ewald && ewald_alpha > 0.0) ? pairs_excl : nullptr;
  c.nexcl = (ewald && ewald_alpha > 0.0 && pairs_excl) ? npairs_excl : 0;
  c.k = prefactor; c.rc = cutoff; c.alpha = ewald ? ewald_alpha : 0.0;
  c.energy = energy; c.e_scale = 1.0;
  c.gx = grad_coords; c.gx_scale = 1.0;
  c.gq = grad_charges;
  c.ws = workspace; c.ws_bytes = workspace_bytes;
  return run_pairs_any(c, (cudaStream_t)stream);
}

}  // extern "C"
