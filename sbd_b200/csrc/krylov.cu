// Vector kernels of the Davidson solvers, without a host round trip inside a
// step.
//
// A step used to read every overlap and norm back (2 ib + 6 waits), with a
// reduction in two launches and an update in a third for each.  Here a
// reduction leaves its block sums in device memory and the next kernel's
// blocks finish it themselves (a fixed order, the same in every block), so
// that one pass per basis vector does the update by the previous overlap and
// the dot product with the next vector:
//
//   correction + <C_0|x>                                1 pass
//   x -= <C_k|x> C_k, then <C_k+1|x> (at last <x|x>)    1 pass per vector
//   x /= |x|                                            1 pass
//   <C_j|HC> for every j                                y read once per 8 vectors
//   W, R, <W|W>, <R|R>                                  1 pass; both scaled in 1
//
// All are HBM bound: modified Gram-Schmidt reads x and two basis vectors and
// writes x per pass, 32 bytes per element instead of 40, and no pass waits for
// the host.  A 10-step FP64 Davidson on 490,000 determinants took 21 ms with
// 4 ms of kernels.
#include <algorithm>
#include <utility>

#include "internal.cuh"

namespace sbdgpu {

namespace {

constexpr int kT = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sum over the block, in every thread
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[kT / 32];
  v = warp_sum(v);
  __syncthreads();  // an earlier sum's values are read
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < kT / 32; w++) s += sh[w];
  return s;
}

// the reduction whose block sums are part[0 .. np)
__device__ __forceinline__ double finish(const double* __restrict__ part, int np) {
  double v = 0.0;
  for (int i = threadIdx.x; i < np; i += kT) v += part[i];
  return block_sum(v);
}

__device__ __forceinline__ void leave(double v, double* __restrict__ part) {
  v = block_sum(v);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// C_new = R / (E0 - H_ii), regularised as davidson.h:855-862, and <C_0|C_new>
template <typename B>
__global__ void __launch_bounds__(kT) correction_kernel(const double* __restrict__ R, const double* __restrict__ hii,
                                                       double e0, const double* __restrict__ e0_dev, double eps_reg,
                                                       double* __restrict__ x, const B* __restrict__ c0, size_t n,
                                                       double* __restrict__ part) {
  if (e0_dev) e0 = *e0_dev;
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * kT + threadIdx.x; i < n; i += (size_t)gridDim.x * kT) {
    const double den = e0 - hii[i];
    const double v = fabs(den) > eps_reg ? R[i] / den : R[i] / (den - eps_reg);
    x[i] = v;
    acc += (double)c0[i] * v;
  }
  leave(acc, part);
}

// block sums of <c|x>
template <typename B>
__global__ void __launch_bounds__(kT) overlap_kernel(const double* __restrict__ x, const B* __restrict__ c, size_t n,
                                                    double* __restrict__ part) {
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * kT + threadIdx.x; i < n; i += (size_t)gridDim.x * kT)
    acc += (double)c[i] * x[i];
  leave(acc, part);
}

// x -= <C|x> C with the overlap's block sums in `in`, then the block sums of
// <next|x> (next null: of <x|x>)
template <typename B>
__global__ void __launch_bounds__(kT) gram_schmidt_kernel(double* __restrict__ x, const B* __restrict__ c,
                                                         const B* __restrict__ next, size_t n,
                                                         const double* __restrict__ in, double* __restrict__ out) {
  const double d = -finish(in, gridDim.x);
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * kT + threadIdx.x; i < n; i += (size_t)gridDim.x * kT) {
    const double v = x[i] + (double)c[i] * d;
    x[i] = v;
    acc += next ? (double)next[i] * v : v * v;
  }
  leave(acc, out);
}

// out = x / sqrt(sum of part)
template <typename B>
__global__ void __launch_bounds__(kT) normalise_kernel(const double* x, B* out, size_t n,
                                                      const double* __restrict__ part) {
  const double a = 1.0 / sqrt(finish(part, gridDim.x));
  for (size_t i = (size_t)blockIdx.x * kT + threadIdx.x; i < n; i += (size_t)gridDim.x * kT) out[i] = (B)(x[i] * a);
}

// block sums of <c_j|y>, j < k <= 8, at part[j * gridDim.x]
template <typename B>
__global__ void __launch_bounds__(kT) dots_kernel(BasisPack<B> c, int first, int k, const B* __restrict__ y, size_t n,
                                                 double* __restrict__ part) {
  double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (size_t i = (size_t)blockIdx.x * kT + threadIdx.x; i < n; i += (size_t)gridDim.x * kT) {
    const double v = (double)y[i];
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j < k) acc[j] += (double)c.p[first + j][i] * v;
  }
#pragma unroll
  for (int j = 0; j < 8; j++)
    if (j < k) leave(acc[j], part + (size_t)j * gridDim.x);
}

// out[j] = sum of part[j * np .. (j + 1) * np), one block per j
__global__ void __launch_bounds__(kT) finish_kernel(const double* __restrict__ part, int np, double* __restrict__ out) {
  const double s = finish(part + (size_t)blockIdx.x * np, np);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// W = sum_k u_k C_k, R = E0 W - sum_k u_k HC_k (davidson.h:772-797) and the
// block sums of <W|W> and <R|R>; u and E0 by value or from device memory
template <typename B>
__global__ void __launch_bounds__(kT) ritz_kernel(BasisPack<B> c, BasisPack<B> hc, int nk, RitzCoef u,
                                                 const double* __restrict__ u_dev, const double* __restrict__ e0_dev,
                                                 double* __restrict__ W, double* __restrict__ R, size_t n,
                                                 double* __restrict__ part_w, double* __restrict__ part_r) {
  __shared__ double su[32];
  if ((int)threadIdx.x < nk) su[threadIdx.x] = u_dev ? u_dev[threadIdx.x] : u.u[threadIdx.x];
  const double e0 = e0_dev ? *e0_dev : u.e0;
  __syncthreads();
  double aw = 0.0, ar = 0.0;
  for (size_t i = (size_t)blockIdx.x * kT + threadIdx.x; i < n; i += (size_t)gridDim.x * kT) {
    double w = 0.0, r = 0.0;
    for (int k = 0; k < nk; k++) {
      w += (double)c.p[k][i] * su[k];
      r -= (double)hc.p[k][i] * su[k];
    }
    r += e0 * w;
    W[i] = w;
    R[i] = r;
    aw += w * w;
    ar += r * r;
  }
  leave(aw, part_w);
  leave(ar, part_r);
}

// W and R divided by their norms; *tol = |R|
__global__ void __launch_bounds__(kT) ritz_scale_kernel(double* __restrict__ W, double* __restrict__ R, size_t n,
                                                       const double* __restrict__ part_w,
                                                       const double* __restrict__ part_r, double* __restrict__ tol) {
  const double w = 1.0 / sqrt(finish(part_w, gridDim.x));
  const double rn = sqrt(finish(part_r, gridDim.x)), r = 1.0 / rn;
  if (blockIdx.x == 0 && threadIdx.x == 0) *tol = rn;
  for (size_t i = (size_t)blockIdx.x * kT + threadIdx.x; i < n; i += (size_t)gridDim.x * kT) {
    W[i] *= w;
    R[i] *= r;
  }
}

unsigned blocks(size_t n) { return (unsigned)std::max<size_t>(1, std::min<size_t>((n + kT - 1) / kT, kKrylovBlocks)); }

}  // namespace

// x = R / (E0 - H_ii) (E0 by value, or from e0_dev; R null: x as it is),
// orthogonalised against C[0 .. k) by modified Gram-Schmidt in `passes` passes
// and normalised into out (which may be x).  part: 32 kKrylovBlocks doubles.
template <typename B>
void krylov_correction(const double* R, const double* hii, double e0, const double* e0_dev, double* x,
                       const B* const* C, int k, B* out, size_t n, int passes, double* part, cudaStream_t s) {
  const unsigned g = blocks(n);
  double* a = part;
  double* b = part + kKrylovBlocks;
  if (R)
    correction_kernel<B><<<g, kT, 0, s>>>(R, hii, e0, e0_dev, 1.0e-12, x, C[0], n, a);
  else
    overlap_kernel<B><<<g, kT, 0, s>>>(x, C[0], n, a);
  for (int pass = 0; pass < passes; pass++)
    for (int j = 0; j < k; j++) {
      const B* next = j + 1 < k ? C[j + 1] : pass + 1 < passes ? C[0] : nullptr;
      gram_schmidt_kernel<B><<<g, kT, 0, s>>>(x, C[j], next, n, a, b);
      std::swap(a, b);
    }
  normalise_kernel<B><<<g, kT, 0, s>>>(x, out, n, a);
  SBD_CUDA(cudaGetLastError());
}

// out[j] = <C_j|y>, j < k <= 32
template <typename B>
void krylov_dots(const B* const* C, int k, const B* y, size_t n, double* part, double* out, cudaStream_t s) {
  const unsigned g = blocks(n);
  BasisPack<B> p{};
  for (int j = 0; j < k; j++) p.p[j] = C[j];
  for (int j = 0; j < k; j += 8)
    dots_kernel<B><<<g, kT, 0, s>>>(p, j, std::min(8, k - j), y, n, part + (size_t)j * g);
  finish_kernel<<<(unsigned)k, kT, 0, s>>>(part, (int)g, out);
  SBD_CUDA(cudaGetLastError());
}

// Ritz vector W and residual R of the coefficients u (by value, or u_dev and
// e0_dev), both normalised; *tol = the residual's norm (device memory)
template <typename B>
void krylov_ritz(const B* const* C, const B* const* HC, int nk, const RitzCoef& u, const double* u_dev,
                 const double* e0_dev, double* W, double* R, size_t n, double* part, double* tol, cudaStream_t s) {
  const unsigned g = blocks(n);
  BasisPack<B> pc{}, ph{};
  for (int k = 0; k < nk; k++) {
    pc.p[k] = C[k];
    ph.p[k] = HC[k];
  }
  ritz_kernel<B><<<g, kT, 0, s>>>(pc, ph, nk, u, u_dev, e0_dev, W, R, n, part, part + kKrylovBlocks);
  ritz_scale_kernel<<<g, kT, 0, s>>>(W, R, n, part, part + kKrylovBlocks, tol);
  SBD_CUDA(cudaGetLastError());
}

#define SBD_KRYLOV(B)                                                                                               \
  template void krylov_correction<B>(const double*, const double*, double, const double*, double*, const B* const*, \
                                     int, B*, size_t, int, double*, cudaStream_t);                                  \
  template void krylov_dots<B>(const B* const*, int, const B*, size_t, double*, double*, cudaStream_t);             \
  template void krylov_ritz<B>(const B* const*, const B* const*, int, const RitzCoef&, const double*, const double*, \
                               double*, double*, size_t, double*, double*, cudaStream_t);
SBD_KRYLOV(double)
SBD_KRYLOV(float)

}  // namespace sbdgpu
