// Neighbour lists: the drop-in kernels behind build_neighbor_list_nsquared(_out) and
// build_neighbor_list_cell_list(_out).
//
// Output contract (both): pairs (cap, 2) int64 filled with -1, found pairs written as
// (larger index, smaller index) in arbitrary order, *npairs = number found (may exceed cap).
//
// Both emit 32x32 tiles of atoms, one warp per work item of up to kEmitTiles tiles of one
// 32-atom group I: every lane tests its atom of I against the atoms of a tile into a 32-bit mask,
// exclusions clear bits, and the item's pairs are compacted lane after lane (an atom's pairs
// lie together, which is what the pair kernels sum over) and written as coalesced 16-byte rows
// behind one global atomic per item. The order of items in the output is not deterministic; the
// SET is. Only the rows after the found pairs are filled with -1 afterwards.
#include <climits>

#include "cluster.cuh"

namespace tff {
namespace {

constexpr int kEmitTiles = kItemTiles;  // tiles per work item (the neighbour search's items)
constexpr int kEmitBlock = 128;
constexpr int kPairCounter = 8;  // status word that counts the pairs of a cell-list build
constexpr int kEmitWarps = kEmitBlock / kWarp;
constexpr int kEmitCodes = 2048;  // staged pairs per item; a denser item is written without staging

// Per-warp staging of an item.
template <class T>
struct EmitSmem {
  typename V4<T>::type pos[kWarp];       // atoms of the current tile
  int idx[kEmitTiles][kWarp];            // caller index of every tile's atoms
  int iidx[kWarp];                       // caller index of I's atoms
  unsigned short code[kEmitCodes];       // lane of I << 7 | tile << 5 | atom of the tile
};

// Where found pairs go. `wide`: rows are 16-byte aligned.
struct EmitOut {
  int64_t *pairs;
  int64_t cap;
  int32_t *counter;
  bool wide;
  __device__ __forceinline__ void put(int64_t row, int a, int b) const {
    if (row >= cap) return;
    const int64_t hi = max(a, b), lo = min(a, b);
    if (wide) {
      reinterpret_cast<longlong2 *>(pairs)[row] = make_longlong2(hi, lo);
    } else {
      pairs[2 * row] = hi;
      pairs[2 * row + 1] = lo;
    }
  }
};

// Writes the pairs of an item: lane l's atom of I with the atoms of tile t whose bit is set in
// m[t]. Called by the whole warp; idx / iidx hold the caller indices.
template <class T>
__device__ __forceinline__ void emit_item(EmitSmem<T> &sm, const unsigned (&m)[kEmitTiles], const EmitOut &out,
                                          int lane) {
  int cnt = 0;
#pragma unroll
  for (int t = 0; t < kEmitTiles; ++t) cnt += __popc(m[t]);
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  const int total = __shfl_sync(kFull, incl, kWarp - 1);
  if (total == 0) return;
  int start = 0;
  if (lane == 0) start = atomicAdd(out.counter, total);
  const int64_t row0 = (unsigned)__shfl_sync(kFull, start, 0);  // counts run to 2^32
  const bool staged = total <= kEmitCodes;
  int at = incl - cnt;
  __syncwarp();
#pragma unroll
  for (int t = 0; t < kEmitTiles; ++t) {
    unsigned mm = m[t];
    while (mm) {
      const int s = __ffs(mm) - 1;
      mm &= mm - 1u;
      if (staged)
        sm.code[at] = (unsigned short)(lane << 7 | t << 5 | s);
      else
        out.put(row0 + at, sm.iidx[lane], sm.idx[t][s]);
      ++at;
    }
  }
  __syncwarp();
  if (staged)
    for (int k = lane; k < total; k += kWarp) {
      const int c = sm.code[k];
      out.put(row0 + k, sm.iidx[c >> 7], sm.idx[(c >> 5) & 3][c & 31]);
    }
  __syncwarp();
}

// FP64 re-test of a candidate pair from the caller's (unwrapped) coordinates, with the
// same minimum-image arithmetic as the FP64 path.
template <class T>
__device__ __forceinline__ bool within_fp64(const T *x, int64_t i, int64_t j, const double *m, const double *inv,
                                            bool periodic, double rc2) {
  double dx = (double)x[3 * i] - (double)x[3 * j];
  double dy = (double)x[3 * i + 1] - (double)x[3 * j + 1];
  double dz = (double)x[3 * i + 2] - (double)x[3 * j + 2];
  if (periodic) min_image(dx, dy, dz, m, inv);
  return dx * dx + dy * dy + dz * dz <= rc2;
}

// Squared distances this close to rc^2 (relative) are decided in FP64 from the caller's
// coordinates when they were computed in FP32.
constexpr float kEdge = 1e-5f;

// All pairs: groups are 32 consecutive atoms; item (I, c) takes the groups p c .. p c + p - 1 up to
// I, p tiles per item (at most kEmitTiles; fewer for small systems, whose items would not fill
// the SMs: 648 atoms FP64 30 -> 10.8 us with single tiles). Items are numbered by rows of p groups I
// that have equally many.
template <class T>
__global__ void __launch_bounds__(kEmitBlock) nsquared_kernel(const T *x, const T *box, int64_t n, double rc,
                                                              const int64_t *row_ptr, const int64_t *col,
                                                              int include_self, EmitOut out, int64_t nitems, int per_item) {
  __shared__ EmitSmem<T> s_emit[kEmitWarps];
  __shared__ double s_m[9], s_inv[9];
  __shared__ T s_mt[9], s_invt[9];
  const bool periodic = box != nullptr;
  if (threadIdx.x == 0 && periodic) {
    Box b;
    load_box(box, b);
    for (int k = 0; k < 9; ++k) {
      s_m[k] = b.m[k];
      s_inv[k] = b.inv[k];
      s_mt[k] = (T)b.m[k];
      s_invt[k] = (T)b.inv[k];
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  EmitSmem<T> &sm = s_emit[w];
  const double rc2 = rc * rc;
  const T rc2t = (T)rc2, edge = sizeof(T) == 4 ? T(kEdge) * rc2t : T(0);
  for (int64_t item = (int64_t)blockIdx.x * kEmitWarps + w; item < nitems; item += (int64_t)gridDim.x * kEmitWarps) {
    // groups pQ .. pQ + p - 1 have Q + 1 items each: p Q (Q + 1) / 2 items come before group pQ
    const auto before = [&](int64_t Q) { return per_item * (Q * (Q + 1) / 2); };
    int64_t Q = (int64_t)floor((sqrt(8.0 * (double)item / per_item + 1.0) - 1.0) * 0.5);
    while (before(Q) > item) --Q;
    while (before(Q + 1) <= item) ++Q;
    const int64_t rest = item - before(Q);
    const int64_t I = per_item * Q + rest / (Q + 1), J0 = per_item * (rest % (Q + 1));
    const int64_t i = I * kWarp + lane;
    const bool iv = i < n;
    T xi = T(0), yi = T(0), zi = T(0);
    if (iv) {
      xi = x[3 * i];
      yi = x[3 * i + 1];
      zi = x[3 * i + 2];
    }
    sm.iidx[lane] = (int)i;
    unsigned m[kEmitTiles] = {};
#pragma unroll
    for (int t = 0; t < kEmitTiles; ++t) {
      const int64_t J = J0 + t;
      if (t >= per_item || J > I) break;
      const int64_t jl = J * kWarp + lane;
      const int nj = (int)min((int64_t)kWarp, n - J * kWarp);
      __syncwarp();
      if (jl < n) sm.pos[lane] = make_v4(x[3 * jl], x[3 * jl + 1], x[3 * jl + 2], T(0));
      sm.idx[t][lane] = (int)jl;
      __syncwarp();
      unsigned in = 0u, near = 0u;
#pragma unroll 4
      for (int s = 0; s < nj; ++s) {
        const auto p = sm.pos[s];
        T dx = xi - p.x, dy = yi - p.y, dz = zi - p.z;
        if (periodic) min_image(dx, dy, dz, s_mt, s_invt);
        const T r2 = dx * dx + dy * dy + dz * dz;
        if (sizeof(T) == 8) {
          in |= r2 <= rc2t ? 1u << s : 0u;
        } else {
          in |= r2 < rc2t - edge ? 1u << s : 0u;
          near |= r2 >= rc2t - edge && r2 <= rc2t + edge ? 1u << s : 0u;
        }
      }
      unsigned ok = iv ? kFull : 0u;
      if (J == I) ok &= include_self ? (2u << lane) - 1u : (1u << lane) - 1u;
      in &= ok;
      near &= ok;
      while (near) {
        const int s = __ffs(near) - 1;
        near &= near - 1u;
        if (within_fp64(x, i, J * kWarp + s, s_m, s_inv, periodic, rc2)) in |= 1u << s;
      }
      if (col && in)
        for (int64_t e = row_ptr[i]; e < row_ptr[i + 1]; ++e) {
          const int64_t d = col[e] - J * kWarp;
          if (d >= 0 && d < kWarp) in &= ~(1u << d);
        }
      m[t] = in;
    }
    emit_item(sm, m, out, lane);
  }
}

// Cell list: items of the neighbour search (cluster I and list entries k, k + n, ... of its n
// items), found through the item offsets.
//
// The mask loop visits only the atoms of J within the cutoff of I's bounding box (two fifths of
// them at rc = 1 nm). Excluded partners are looked up by their slot, and only for tiles in the
// range of clusters that hold a partner of I's atoms. 9,000 atoms, 1.9 M pairs: 114 -> 41 us against
// a push per tested pair with a row search per hit (and 7 us less of filling rows).
template <class T>
__global__ void __launch_bounds__(kEmitBlock) cell_emit_kernel(ClusterData<T> d, const T *x, double rc,
                                                               const int64_t *row_ptr, const int64_t *col,
                                                               int include_self, EmitOut out) {
  pdl_enter();
  using V = typename V4<T>::type;
  __shared__ EmitSmem<T> s_emit[kEmitWarps];
  __shared__ double s_info[kInfoStride];
  __shared__ T s_mt[9], s_invt[9];
  if (threadIdx.x < kInfoStride) s_info[threadIdx.x] = d.boxinfo[threadIdx.x];
  if (threadIdx.x < 9) {
    s_mt[threadIdx.x] = (T)d.boxinfo[threadIdx.x];
    s_invt[threadIdx.x] = (T)d.boxinfo[9 + threadIdx.x];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  EmitSmem<T> &sm = s_emit[w];
  const double rc2 = rc * rc;
  const T rc2t = (T)rc2, edge = sizeof(T) == 4 ? T(kEdge) * rc2t : T(0);
  const T Lx = s_mt[0], Ly = s_mt[4], Lz = s_mt[8];
  const T iLx = s_invt[0], iLy = s_invt[4], iLz = s_invt[8];
  const bool ortho = s_info[18] != 0.0;
  // a 1e-5 wider cutoff for the atom-to-box test keeps what the distance test's edge may keep
  const double rc_box = rc * (1.0 + 1e-5);
  BoxTestF bt{};
  if constexpr (sizeof(T) == 4) bt = box_test_f(s_info, rc_box);
  const int ncl = (int)d.nclusters;
  const int nitems = d.itemoff[ncl];
  for (int item = blockIdx.x * kEmitWarps + w; item < nitems; item += gridDim.x * kEmitWarps) {
    const int I = item_cluster(d.itemoff, ncl, item);
    const int k0 = item - d.itemoff[I], n = d.itemoff[I + 1] - d.itemoff[I], cnt = d.ncount[I];
    const int64_t si = (int64_t)I * kWarp + lane;
    const int ai = d.sidx[si];
    const V pi = d.pos[si], ci = d.bc[I], hi = d.bh[I];
    const V zero = make_v4(T(0), T(0), T(0), T(0));
    sm.iidx[lane] = ai;
    // exclusion row of the lane's atom and the warp's range of partner clusters
    int64_t e0 = 0, e1 = 0;
    int x_lo = INT_MAX, x_hi = -1;
    if (col && ai >= 0) {
      e0 = row_ptr[ai];
      e1 = row_ptr[ai + 1];
      for (int64_t e = e0; e < e1; ++e) {
        const int64_t c = col[e];
        if (c < 0 || c >= d.natoms) continue;
        const int J = d.inv[c] >> 5;
        x_lo = min(x_lo, J);
        x_hi = max(x_hi, J);
      }
    }
    x_lo = __reduce_min_sync(kFull, x_lo);
    x_hi = __reduce_max_sync(kFull, x_hi);
    unsigned m[kEmitTiles] = {};
#pragma unroll
    for (int t = 0; t < kEmitTiles; ++t) {
      if (k0 + t * n >= cnt) break;
      const int J = d.nbr[(int64_t)I * d.cap + k0 + t * n];
      const int64_t sj = (int64_t)J * kWarp + lane;
      const int aj = d.sidx[sj];
      const V f = d.frac[sj];
      __syncwarp();
      sm.pos[lane] = d.pos[sj];
      sm.idx[t][lane] = aj;
      bool reach;
      if constexpr (sizeof(T) == 4)
        reach = boxes_may_interact_f(ci, hi, f, zero, bt);
      else
        reach = clusters_may_interact<T>(ci, hi, f, zero, s_info, rc_box);
      unsigned left = __ballot_sync(kFull, aj >= 0 && reach);
      __syncwarp();
      unsigned in = 0u, near = 0u;
      while (left) {
        const int s = __ffs(left) - 1;
        left &= left - 1u;
        const V p = sm.pos[s];
        T dx = pi.x - p.x, dy = pi.y - p.y, dz = pi.z - p.z;
        if (ortho) {
          dx = wrap1(dx, Lx, iLx);
          dy = wrap1(dy, Ly, iLy);
          dz = wrap1(dz, Lz, iLz);
        } else {
          min_image(dx, dy, dz, s_mt, s_invt);
        }
        const T r2 = dx * dx + dy * dy + dz * dz;
        if (sizeof(T) == 8) {
          in |= r2 <= rc2t ? 1u << s : 0u;
        } else {
          in |= r2 < rc2t - edge ? 1u << s : 0u;
          near |= r2 >= rc2t - edge && r2 <= rc2t + edge ? 1u << s : 0u;
        }
      }
      unsigned ok = ai >= 0 ? kFull : 0u;
      if (J == I) ok &= include_self ? (2u << lane) - 1u : (1u << lane) - 1u;
      in &= ok;
      near &= ok;
      while (near) {
        const int s = __ffs(near) - 1;
        near &= near - 1u;
        if (within_fp64(x, ai, sm.idx[t][s], s_info, s_info + 9, true, rc2)) in |= 1u << s;
      }
      if (J >= x_lo && J <= x_hi && in)
        for (int64_t e = e0; e < e1; ++e) {
          const int64_t c = col[e];
          if (c < 0 || c >= d.natoms) continue;
          const int slot = d.inv[c];
          if ((slot >> 5) == J) in &= ~(1u << (slot & 31));
        }
      m[t] = in;
    }
    emit_item(sm, m, out, lane);
  }
}

// Fills rows [count, cap) with -1 and reports the count: *npairs = count, or INT_MAX when a
// cluster's neighbour list overflowed (the caller sees npairs > cap).
__global__ void __launch_bounds__(256) pad_rows_kernel(const int32_t *count, const unsigned *status, int64_t *pairs,
                                                       int64_t cap, int32_t *npairs) {
  pdl_enter();
  const int32_t found = *count;
  for (int64_t k = 2 * (int64_t)(unsigned)found + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < 2 * cap;
       k += (int64_t)gridDim.x * blockDim.x)
    pairs[k] = -1;
  if (blockIdx.x == 0 && threadIdx.x == 0 && status) npairs[0] = (status[0] & 1u) ? INT_MAX : found;
}

int default_cluster_cap(int64_t nclusters, int requested) {
  if (requested > 0) return requested;
  return (int)std::max<int64_t>(1, std::min<int64_t>(nclusters, 1024));
}

int launch_pad(const int32_t *count, const unsigned *status, int64_t *pairs, int64_t cap, int32_t *npairs,
               cudaStream_t s) {
  const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((2 * cap + 255) / 256, (int64_t)sm_count() * 8));
  return launch_k(true, pad_rows_kernel, nb, 256, 0, s, count, status, pairs, cap, npairs);
}

bool rows_aligned(const int64_t *pairs) { return (reinterpret_cast<uintptr_t>(pairs) & 15) == 0; }

template <class T>
int nsquared_impl(int64_t natoms, const T *x, const T *box, double cutoff, const int64_t *rp,
                  const int64_t *col, int include_self, int64_t *pairs, int64_t cap, int32_t *npairs,
                  cudaStream_t s) {
  TFF_CUDA(cudaMemsetAsync(npairs, 0, sizeof(int32_t), s));
  if (natoms > 0) {
    const int64_t groups = (natoms + kWarp - 1) / kWarp;
    // one tile per item until there are several warps of them for every SM
    const int per = (int)std::max<int64_t>(1, std::min<int64_t>(kEmitTiles, groups * groups / 2 / (16 * sm_count())));
    const int64_t q = groups / per, r = groups % per, items = per * (q * (q + 1) / 2) + r * (q + 1);
    const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((items + kEmitWarps - 1) / kEmitWarps,
                                                               (int64_t)sm_count() * 16));
    const EmitOut out{pairs, cap, npairs, rows_aligned(pairs)};
    nsquared_kernel<T><<<nb, kEmitBlock, 0, s>>>(x, box, natoms, cutoff, rp, col, include_self, out, items, per);
    TFF_LAUNCHED();
  }
  return cap > 0 ? launch_pad(npairs, nullptr, pairs, cap, npairs, s) : TFF_OK;
}

template <class T>
int cell_list_impl(int64_t natoms, const T *x, const T *box, double cutoff, const int64_t *rp, const int64_t *col,
                   int include_self, int64_t *pairs, int64_t cap, int32_t *npairs, int ccap, void *ws,
                   size_t ws_bytes, cudaStream_t s) {
  const int dtype = sizeof(T) == 8 ? TFF_F64 : TFF_F32;
  const int64_t ncl = (natoms + kWarp - 1) / kWarp;
  ClusterLayout L = cluster_layout(dtype, natoms, default_cluster_cap(ncl, ccap), false);
  if (ws == nullptr || ws_bytes < L.bytes) {
    set_error("workspace too small: need %zu bytes, got %zu", L.bytes, ws_bytes);
    return TFF_ERR_WORKSPACE;
  }
  if (natoms == 0) {
    if (cap > 0) TFF_CUDA(cudaMemsetAsync(pairs, 0xff, sizeof(int64_t) * 2 * cap, s));
    TFF_CUDA(cudaMemsetAsync(npairs, 0, sizeof(int32_t), s));
    return TFF_OK;
  }
  ClusterData<T> d = cluster_data<T>(L, ws);
  int st = build_clusters<T>(L, d, ws, x, nullptr, box, cutoff, /*half=*/1, s, nullptr, 0, /*pdl=*/true);
  if (st != TFF_OK) return st;
  // the pair counter is a status word of the build (cleared with them)
  const EmitOut out{pairs, cap, reinterpret_cast<int32_t *>(d.status + kPairCounter), rows_aligned(pairs)};
  const int64_t items = item_capacity(L.nclusters, L.cap);
  const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((items + kEmitWarps - 1) / kEmitWarps,
                                                             (int64_t)sm_count() * 16));
  st = launch_k(true, cell_emit_kernel<T>, nb, kEmitBlock, 0, s, d, x, cutoff, rp, col, include_self, out);
  if (st != TFF_OK) return st;
  return launch_pad(out.counter, d.status, pairs, cap, npairs, s);
}

}  // namespace
}  // namespace tff

using namespace tff;

extern "C" {

int tff_nblist_nsquared(int dtype, int64_t natoms, const void *coords, const void *box, double cutoff,
                        const int64_t *excl_row_ptr, const int64_t *excl_col, int include_self, int64_t *pairs,
                        int64_t max_npairs, int32_t *npairs, tff_stream_t stream) {
  TFF_NVTX("tff_nblist_nsquared");
  TFF_ARG(dtype == TFF_F32 || dtype == TFF_F64, "dtype must be TFF_F32 or TFF_F64");
  TFF_ARG(natoms >= 0 && max_npairs >= 0, "negative sizes");
  TFF_ARG(npairs != nullptr, "npairs is NULL");
  TFF_ARG(pairs != nullptr || max_npairs == 0, "pairs is NULL");
  TFF_ARG(coords != nullptr || natoms == 0, "coords is NULL");
  TFF_ARG((excl_row_ptr == nullptr) == (excl_col == nullptr), "exclusion CSR needs both arrays");
  TFF_ARG(cutoff >= 0.0, "cutoff must be >= 0");
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TFF_F32)
    return nsquared_impl<float>(natoms, (const float *)coords, (const float *)box, cutoff, excl_row_ptr, excl_col,
                                include_self, pairs, max_npairs, npairs, s);
  return nsquared_impl<double>(natoms, (const double *)coords, (const double *)box, cutoff, excl_row_ptr, excl_col,
                               include_self, pairs, max_npairs, npairs, s);
}

size_t tff_nblist_cell_list_workspace_bytes(int dtype, int64_t natoms, int max_cluster_neighbors) {
  const int64_t ncl = (natoms + kWarp - 1) / kWarp;
  return cluster_layout(dtype, natoms, default_cluster_cap(ncl, max_cluster_neighbors), false).bytes;
}

int tff_nblist_cell_list(int dtype, int64_t natoms, const void *coords, const void *box, double cutoff,
                         const int64_t *excl_row_ptr, const int64_t *excl_col, int include_self, int64_t *pairs,
                         int64_t max_npairs, int32_t *npairs, int max_cluster_neighbors, void *workspace,
                         size_t workspace_bytes, tff_stream_t stream) {
  TFF_NVTX("tff_nblist_cell_list");
  TFF_ARG(dtype == TFF_F32 || dtype == TFF_F64, "dtype must be TFF_F32 or TFF_F64");
  TFF_ARG(box != nullptr, "Cell-list neighbor list requires a periodic box");
  TFF_ARG(natoms >= 0 && max_npairs >= 0, "negative sizes");
  TFF_ARG(npairs != nullptr, "npairs is NULL");
  TFF_ARG(pairs != nullptr || max_npairs == 0, "pairs is NULL");
  TFF_ARG(coords != nullptr || natoms == 0, "coords is NULL");
  TFF_ARG((excl_row_ptr == nullptr) == (excl_col == nullptr), "exclusion CSR needs both arrays");
  TFF_ARG(cutoff >= 0.0, "cutoff must be >= 0");
  TFF_ARG(natoms < (int64_t)INT_MAX, "too many atoms");
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == TFF_F32)
    return cell_list_impl<float>(natoms, (const float *)coords, (const float *)box, cutoff, excl_row_ptr, excl_col,
                                 include_self, pairs, max_npairs, npairs, max_cluster_neighbors, workspace,
                                 workspace_bytes, s);
  return cell_list_impl<double>(natoms, (const double *)coords, (const double *)box, cutoff, excl_row_ptr, excl_col,
                                include_self, pairs, max_npairs, npairs, max_cluster_neighbors, workspace,
                                workspace_bytes, s);
}

}  // extern "C"
