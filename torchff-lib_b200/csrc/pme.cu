// PME entry points: plan management and the drop-in pme_long_range (rank 0).
#include <algorithm>
#include <cmath>
#include <vector>

#include "pme.cuh"

namespace tff {

int pme_cufft_fail(cufftResult r, const char *what) {
  set_error("cuFFT error %d in %s", (int)r, what);
  return TFF_ERR_CUFFT;
}

namespace {

// The three launches of a solve over planes (pme_fft.cuh), programmatic dependents of the kernel
// before: a kernel copies its tables (and works out its influence function) while that one ends; no
// kernel of the chain writes tables, box or moduli, and the forward kernel lets the solve start only after
// its own wait, so whatever wrote the box has completed by then (the rule of launch_k).
// A block lets the next kernel start only when it has nothing but its result left to write, so
// that waiting blocks do not sit on SMs that the real-space stream could use. The solve's blocks
// split a row's kz range so that small grids use every SM.
//
// Bound by latency: a plane is 4-6 short phases between barriers, on K (solve: up to 148) SMs.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class T>
constexpr int kFftMinBlocks = sizeof(T) == 4 ? 3 : 2;  // registers: 80 and 122 of a thread

template <class T>
__global__ void __launch_bounds__(kFftThreads, kFftMinBlocks<T>)
    pme_fft_forward_kernel(const typename Acc<T>::S *grid, Cplx<T> *spec, int K, const Cplx<T> *tables) {
  FftPlan f = fft_plan<T>(K, tables);
  const int64_t x = blockIdx.x;
  wait_for_previous();
  fft_forward_plane<T>(f, grid + x * K * K, spec + x * K * (K / 2 + 1), [] { let_next_start(); });
}

template <class T>
__global__ void __launch_bounds__(kFftThreads, kFftMinBlocks<T>)
    pme_fft_solve_kernel(Cplx<T> *spec, int K, const Cplx<T> *tables, int chunk, const T *box, double alpha,
                         const T *xmod, const T *ymod, const T *zmod, double *partials, unsigned *ticket,
                         double *e_rec) {
  __shared__ PmeShared sh;
  __shared__ Influence inf;
  if (threadIdx.x == 0) {
    load_pme_shared(box, K, sh);
    load_influence(sh, alpha, inf);
  }
  FftPlan f = fft_plan<T>(K, tables);
  __syncthreads();
  const int ky = blockIdx.x, z0 = blockIdx.y * chunk, z1 = min(z0 + chunk, K / 2 + 1);
  const double e = fft_solve_row<T>(
      f, spec, ky, z0, z1, [&](int ix, int iz) { return influence<T>(inf, K, ix, ky, iz, xmod, ymod, zmod); },
      [] { wait_for_previous(); }, [] { let_next_start(); });
  grid_sum_n<kFftThreads>(0.5 * e, partials, ticket, e_rec, false, blockIdx.y * gridDim.x + blockIdx.x,
                          gridDim.x * gridDim.y);
}

template <class T>
__global__ void __launch_bounds__(kFftThreads, kFftMinBlocks<T>)
    pme_fft_inverse_kernel(const Cplx<T> *spec, T *phi, int K, const Cplx<T> *tables) {
  FftPlan f = fft_plan<T>(K, tables);
  const int64_t x = blockIdx.x;
  wait_for_previous();
  fft_inverse_plane<T>(f, spec + x * K * (K / 2 + 1), phi + x * K * K, [] {});
}

template <class T>
int plane_setup(int K, void **tables) {
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  TFF_CUDA(cudaFuncSetAttribute(pme_fft_forward_kernel<T>, attr, (int)kFftSmemMax));
  TFF_CUDA(cudaFuncSetAttribute(pme_fft_solve_kernel<T>, attr, (int)kFftSmemMax));
  TFF_CUDA(cudaFuncSetAttribute(pme_fft_inverse_kernel<T>, attr, (int)kFftSmemMax));
  std::vector<Cplx<T>> tab;
  fft_table<T>(K, tab);
  TFF_CUDA(cudaMalloc(tables, tab.size() * sizeof(Cplx<T>)));
  cudaError_t e = cudaMemcpy(*tables, tab.data(), tab.size() * sizeof(Cplx<T>), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // other streams do not wait for stream 0
  if (e != cudaSuccess) {
    cudaFree(*tables);
    *tables = nullptr;
    return cuda_fail(e, "transform tables", __FILE__, __LINE__);
  }
  return TFF_OK;
}

// Fixed point -> FP32 for cuFFT.
__global__ void pme_fix_to_real_kernel(const unsigned long long *gi, float *gf, int64_t n) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    gf[k] = (float)from_fix(gi[k]);
}

// Influence function over the whole spectrum (cuFFT path).
template <class T>
__global__ void __launch_bounds__(kPmeBlock) pme_convolve_kernel(typename CplxOf<T>::type *S, const T *box, int K,
                                                                 double alpha, const T *xmod, const T *ymod,
                                                                 const T *zmod, double *partials, unsigned *ticket,
                                                                 double *e_rec) {
  __shared__ PmeShared sh;
  __shared__ Influence inf;
  if (threadIdx.x == 0) {
    load_pme_shared(box, K, sh);
    load_influence(sh, alpha, inf);
  }
  __syncthreads();
  const unsigned Kz = K / 2 + 1, total = (unsigned)K * K * Kz;  // K <= 1024: fits 32 bits
  double e = 0.0;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const unsigned row = t / Kz, x = row / (unsigned)K;
    const int iz = (int)(t - row * Kz);
    const double c = influence<T>(inf, K, (int)x, (int)(row - x * K), iz, xmod, ymod, zmod);
    auto v = S[t];
    const double re = v.x, im = v.y;
    e += (iz == 0 || 2 * iz == K ? 1.0 : 2.0) * c * (re * re + im * im);
    v.x = (T)(re * c);
    v.y = (T)(im * c);
    S[t] = v;
  }
  grid_sum<kPmeBlock>(0.5 * e, partials, ticket, e_rec, false);
}

}  // namespace

template <class T>
int pme_solve_phase(const PmePlanImpl &p, const PmeLayout &L, char *ws, const T *box, double alpha, const T *xmod,
                    const T *ymod, const T *zmod, cudaStream_t s, T **phi_grid, bool after_kernel) {
  using S = typename Acc<T>::S;
  const int K = p.K;
  const int sms = sm_count();
  S *grid = reinterpret_cast<S *>(ws + L.fix);
  T *real = sizeof(T) == 4 ? reinterpret_cast<T *>(ws + L.real) : reinterpret_cast<T *>(grid);
  double *partials = reinterpret_cast<double *>(ws + L.partials);
  unsigned *tickets = reinterpret_cast<unsigned *>(ws + L.tickets);
  double *energies = reinterpret_cast<double *>(ws + L.energies);
  *phi_grid = real;
  if (p.planes) {
    auto *spec = reinterpret_cast<Cplx<T> *>(ws + L.cplx);
    const auto *tables = static_cast<const Cplx<T> *>(p.tables);
    const size_t smem = fft_smem<T>(K);
    // as many parts of a row as keep the blocks within one wave of one per SM
    const int Kz = K / 2 + 1, split = std::min(Kz, std::max(1, sms / K)), chunk = (Kz + split - 1) / split;
    int st = launch_k(after_kernel, pme_fft_forward_kernel<T>, K, kFftThreads, smem, s, static_cast<const S *>(grid),
                      spec, K, tables);
    if (st != TFF_OK) return st;
    st = launch_k(true, pme_fft_solve_kernel<T>, dim3(K, (Kz + chunk - 1) / chunk), kFftThreads, smem, s, spec, K,
                  tables, chunk, box, alpha, xmod, ymod, zmod, partials, tickets, energies);
    if (st != TFF_OK) return st;
    return launch_k(true, pme_fft_inverse_kernel<T>, K, kFftThreads, smem, s, static_cast<const Cplx<T> *>(spec), real,
                    K, tables);
  }
  if (sizeof(T) == 4) {
    const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((L.ngrid + 255) / 256, sms * 8));
    pme_fix_to_real_kernel<<<nb, 256, 0, s>>>(reinterpret_cast<unsigned long long *>(grid),
                                              reinterpret_cast<float *>(real), L.ngrid);
    TFF_LAUNCHED();
  }
  auto *cplx = reinterpret_cast<typename CplxOf<T>::type *>(ws + L.cplx);
  cufftResult r;
  if ((r = cufftSetStream(p.r2c, s)) != CUFFT_SUCCESS) return pme_cufft_fail(r, "cufftSetStream");
  if ((r = cufftSetStream(p.c2r, s)) != CUFFT_SUCCESS) return pme_cufft_fail(r, "cufftSetStream");
  if (sizeof(T) == 4)
    r = cufftExecR2C(p.r2c, reinterpret_cast<cufftReal *>(real), reinterpret_cast<cufftComplex *>(cplx));
  else
    r = cufftExecD2Z(p.r2c, reinterpret_cast<cufftDoubleReal *>(real), reinterpret_cast<cufftDoubleComplex *>(cplx));
  if (r != CUFFT_SUCCESS) return pme_cufft_fail(r, "forward FFT");
  const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((L.ncplx + kPmeBlock - 1) / kPmeBlock, sms * 4));
  pme_convolve_kernel<T><<<nb, kPmeBlock, 0, s>>>(cplx, box, K, alpha, xmod, ymod, zmod, partials, tickets, energies);
  TFF_LAUNCHED();
  if (sizeof(T) == 4)
    r = cufftExecC2R(p.c2r, reinterpret_cast<cufftComplex *>(cplx), reinterpret_cast<cufftReal *>(real));
  else
    r = cufftExecZ2D(p.c2r, reinterpret_cast<cufftDoubleComplex *>(cplx), reinterpret_cast<cufftDoubleReal *>(real));
  if (r != CUFFT_SUCCESS) return pme_cufft_fail(r, "inverse FFT");
  return TFF_OK;
}

template int pme_solve_phase<float>(const PmePlanImpl &, const PmeLayout &, char *, const float *, double, const float *,
                                    const float *, const float *, cudaStream_t, float **, bool);
template int pme_solve_phase<double>(const PmePlanImpl &, const PmeLayout &, char *, const double *, double,
                                     const double *, const double *, const double *, cudaStream_t, double **, bool);

namespace {

template <class T>
int pme_long_range_impl(const PmePlanImpl &p, int64_t n, const T *x, const T *box, const T *q, double alpha,
                        const T *xm, const T *ym, const T *zm, T *energy, T *phi, T *grad, void *ws, size_t ws_bytes,
                        cudaStream_t s) {
  PmeLayout L = pme_layout(p.dtype, p.K);
  if (ws == nullptr || ws_bytes < L.bytes) {
    set_error("workspace too small: need %zu bytes, got %zu", L.bytes, ws_bytes);
    return TFF_ERR_WORKSPACE;
  }
  char *w = static_cast<char *>(ws);
  PlainAtoms<T> atoms{x, q, n};
  T *phi_grid = nullptr;
  int st = pme_grid_phase<T>(p, L, w, atoms, n, box, alpha, xm, ym, zm, s, &phi_grid);
  if (st != TFF_OK) return st;
  if (n == 0) {
    // no atoms: energy is the (zero) reciprocal sum
    TFF_CUDA(cudaMemsetAsync(energy, 0, sizeof(T), s));
    return TFF_OK;
  }
  PlainGatherOut<T> out{phi, grad};
  return pme_gather_phase<T>(p, L, w, atoms, n, box, alpha, phi_grid, out, 1.0, energy, s);
}

}  // namespace
}  // namespace tff

using namespace tff;

extern "C" {

int tff_pme_plan_create(int dtype, int K, tff_pme_plan *plan) {
  TFF_ARG(dtype == TFF_F32 || dtype == TFF_F64, "dtype must be TFF_F32 or TFF_F64");
  TFF_ARG(K >= 6 && K <= 1024, "PME grid K must be in [6, 1024] (order-6 splines)");
  TFF_ARG(plan != nullptr, "plan is NULL");
  auto *p = new tff_pme_plan_s();
  p->impl.dtype = dtype;
  p->impl.K = K;
  cudaGetDevice(&p->impl.device);
  p->impl.planes = fft_planes(K);
  if (p->impl.planes) {
    const int st = dtype == TFF_F64 ? plane_setup<double>(K, &p->impl.tables) : plane_setup<float>(K, &p->impl.tables);
    if (st != TFF_OK) {
      delete p;
      return st;
    }
    *plan = p;
    return TFF_OK;
  }
  cufftResult r = cufftPlan3d(&p->impl.r2c, K, K, K, dtype == TFF_F64 ? CUFFT_D2Z : CUFFT_R2C);
  if (r != CUFFT_SUCCESS) {
    delete p;
    return pme_cufft_fail(r, "cufftPlan3d(R2C)");
  }
  r = cufftPlan3d(&p->impl.c2r, K, K, K, dtype == TFF_F64 ? CUFFT_Z2D : CUFFT_C2R);
  if (r != CUFFT_SUCCESS) {
    cufftDestroy(p->impl.r2c);
    delete p;
    return pme_cufft_fail(r, "cufftPlan3d(C2R)");
  }
  *plan = p;
  return TFF_OK;
}

int tff_pme_plan_destroy(tff_pme_plan plan) {
  if (!plan) return TFF_OK;
  if (plan->impl.planes) {
    cudaFree(plan->impl.tables);
  } else {
    cufftDestroy(plan->impl.r2c);
    cufftDestroy(plan->impl.c2r);
  }
  delete plan;
  return TFF_OK;
}

size_t tff_pme_workspace_bytes(tff_pme_plan plan, int64_t natoms) {
  (void)natoms;
  if (!plan) return 0;
  return pme_layout(plan->impl.dtype, plan->impl.K).bytes;
}

int tff_pme_long_range(tff_pme_plan plan, int64_t natoms, const void *coords, const void *box, const void *charges,
                       double alpha, const void *xmoduli, const void *ymoduli, const void *zmoduli, void *energy,
                       void *phi, void *grad_coords, void *workspace, size_t workspace_bytes, tff_stream_t stream) {
  TFF_NVTX("tff_pme_long_range");
  TFF_ARG(plan != nullptr, "plan is NULL");
  TFF_ARG(natoms >= 0, "negative natoms");
  TFF_ARG(box != nullptr, "PME requires a periodic box");
  TFF_ARG(energy != nullptr, "energy is NULL");
  TFF_ARG(natoms == 0 || (coords != nullptr && charges != nullptr), "coords/charges is NULL");
  TFF_ARG(xmoduli && ymoduli && zmoduli, "B-spline moduli are NULL");
  TFF_ARG(alpha > 0.0, "alpha must be positive");
  cudaStream_t s = (cudaStream_t)stream;
  if (plan->impl.dtype == TFF_F32)
    return pme_long_range_impl<float>(plan->impl, natoms, (const float *)coords, (const float *)box,
                                      (const float *)charges, alpha, (const float *)xmoduli, (const float *)ymoduli,
                                      (const float *)zmoduli, (float *)energy, (float *)phi, (float *)grad_coords,
                                      workspace, workspace_bytes, s);
  return pme_long_range_impl<double>(plan->impl, natoms, (const double *)coords, (const double *)box,
                                     (const double *)charges, alpha, (const double *)xmoduli, (const double *)ymoduli,
                                     (const double *)zmoduli, (double *)energy, (double *)phi, (double *)grad_coords,
                                     workspace, workspace_bytes, s);
}

}  // extern "C"
