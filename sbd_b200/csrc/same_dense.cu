// Same-spin terms of the FP64 sigma as one dense product on the FP64 tensor
// pipe, for bases of some hundreds of strings per spin.
//
// The string-only same-spin operators (the reference's alpha-only and
// beta-only tasks, chemistry/tpb/mult.h:498-566, without the diagonal and the
// singles' Coulomb parts) are 20-70 % dense on such bases, and
//
//   sigma += H0_a C + C H0_b = [ H0_a | C ] [ C ; H0_b ]   (H0_b symmetric)
//
// is one row-major product with K = na + nb: one launch and no transposes.  The
// rows kernels it replaces here stream a row of C per table entry at a seventh
// of the FP64 rate.  CTA tiles of 64 x 64 (32 x 32 for the smallest bases), K
// in steps of 16 through a cp.async ring and dealt to several CTAs that add to
// sigma with atomics, for balance; rows of the staged tiles are padded so that
// the fragments' 8-byte loads hit 16 different bank pairs per half-warp.  Bound
// by the FP64 tensor pipe (69 % busy at 1501 x 803 strings).  Both spins'
// terms, rows kernels -> product: 1501 x 803 strings 0.50 -> 0.25 ms, 495 x 495
// 88 -> 36 us.
//
// A NaN or an infinity times a zero of the dense operator would reach sigma
// entries that no excitation connects: a tile with a non-finite result is
// evaluated again from the excitation tables.
#include <algorithm>
#include <cmath>

#include "device.cuh"
#include "internal.cuh"

namespace sbdgpu {

namespace {

constexpr int kThreads = 128;
constexpr int kBK = 16;

struct Tables {
  const int64_t* s_off;
  const int32_t* s_idx;
  const double* s_val;
  const int64_t* d_off;
  const int32_t* d_idx;
  const double* d_val;
};
Tables view(const SpinTables& t) { return Tables{t.s_off, t.s_idx, t.s_val, t.d_off, t.d_idx, t.d_val}; }

template <int BYTES>
__device__ __forceinline__ void copy_async(double* dst, const double* src, bool on) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = on ? BYTES : 0;  // the rest is zero-filled
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// ROWS x COLS tile of a row-major matrix (ld, rows, cols; row0, col0) into
// dst with row pitch PITCH, zeros outside.  V = 2: ld even, 16-byte aligned
// base, cols even.
template <int ROWS, int COLS, int PITCH, int V>
__device__ __forceinline__ void load_tile(double* dst, const double* __restrict__ src, size_t ld, size_t rows,
                                          size_t cols, size_t row0, size_t col0) {
  constexpr int PER_ROW = COLS / V;
#pragma unroll
  for (int i = threadIdx.x; i < ROWS * PER_ROW; i += kThreads) {
    const int r = i / PER_ROW, c = (i - r * PER_ROW) * V;
    const bool on = row0 + r < rows && col0 + c < cols;
    copy_async<8 * V>(dst + r * PITCH + c, on ? src + (row0 + r) * ld + col0 + c : src, on);
  }
}

// sum over a string's table entries in [lo, hi) of value * x[entry * stride]
__device__ double sparse_dot(const Tables& t, size_t i, const double* __restrict__ x, size_t stride, int64_t lo,
                             int64_t hi) {
  double acc = 0.0;
  for (int64_t k = t.s_off[i]; k < t.s_off[i + 1]; k++)
    if (t.s_idx[k] >= lo && t.s_idx[k] < hi) acc += t.s_val[k] * x[(size_t)t.s_idx[k] * stride];
  for (int64_t k = t.d_off[i]; k < t.d_off[i + 1]; k++)
    if (t.d_idx[k] >= lo && t.d_idx[k] < hi) acc += t.d_val[k] * x[(size_t)t.d_idx[k] * stride];
  return acc;
}

// cp.async stages: deep where a CTA's steps are short
template <int WM, int WN>
__host__ __device__ constexpr int stages() {
  return WM * WN <= 2 ? 6 : 4;
}

// S (na x nb) += H0a C + C H0b; each warp of the 2 x 2 takes (16 WM) x (8 WN).
template <int WM, int WN, int V>
__global__ void __launch_bounds__(kThreads) same_dense_kernel(const double* __restrict__ Ha, size_t lda,
                                                             const double* __restrict__ Hb, size_t ldb,
                                                             const double* __restrict__ C, double* __restrict__ S,
                                                             size_t na, size_t nb, Tables ta, Tables tb) {
  constexpr int BM = 32 * WM, BN = 16 * WN, AP = kBK + 4, BP = BN + 4, kStages = stages<WM, WN>();
  extern __shared__ __align__(16) double smem_d[];
  double* As = smem_d;                       // [stages][BM][AP]
  double* Bs = smem_d + kStages * BM * AP;   // [stages][kBK][BP]
  const size_t row0 = (size_t)blockIdx.y * BM, col0 = (size_t)blockIdx.x * BN;
  const int steps_a = (int)((na + kBK - 1) / kBK), all = steps_a + (int)((nb + kBK - 1) / kBK);
  // this CTA's share of K
  const int first = (int)((int64_t)all * blockIdx.z / gridDim.z);
  const int steps = (int)((int64_t)all * (blockIdx.z + 1) / gridDim.z) - first;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp >> 1) * 16 * WM, wn = (warp & 1) * 8 * WN;
  const int r = lane >> 2, q = lane & 3;
  const auto fetch = [&](int at) {
    if (at < steps) {
      double* a = As + (at % kStages) * BM * AP;
      double* b = Bs + (at % kStages) * kBK * BP;
      const int step = first + at;
      if (step < steps_a) {
        const size_t k0 = (size_t)step * kBK;
        load_tile<BM, kBK, AP, V>(a, Ha, lda, na, V == 2 ? lda : na, row0, k0);
        load_tile<kBK, BN, BP, V>(b, C, nb, na, nb, k0, col0);
      } else {
        const size_t k0 = (size_t)(step - steps_a) * kBK;
        load_tile<BM, kBK, AP, V>(a, C, nb, na, nb, row0, k0);
        load_tile<kBK, BN, BP, V>(b, Hb, ldb, nb, nb, k0, col0);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[WM][WN][4];
#pragma unroll
  for (int i = 0; i < WM; i++)
#pragma unroll
    for (int j = 0; j < WN; j++)
#pragma unroll
      for (int x = 0; x < 4; x++) acc[i][j][x] = 0.0;
#pragma unroll
  for (int s = 0; s < kStages - 1; s++) fetch(s);
  for (int step = 0; step < steps; step++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    fetch(step + kStages - 1);
    const double* a = As + (step % kStages) * BM * AP;
    const double* b = Bs + (step % kStages) * kBK * BP;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double fa[WM][2], fb[WN];
#pragma unroll
      for (int i = 0; i < WM; i++) {
        fa[i][0] = a[(wm + 16 * i + r) * AP + kk + q];
        fa[i][1] = a[(wm + 16 * i + 8 + r) * AP + kk + q];
      }
#pragma unroll
      for (int j = 0; j < WN; j++) fb[j] = b[(kk + q) * BP + wn + 8 * j + r];
#pragma unroll
      for (int i = 0; i < WM; i++)
#pragma unroll
        for (int j = 0; j < WN; j++) mma16(acc[i][j], fa[i][0], fa[i][1], fb[j]);
    }
  }
  bool bad = false;
#pragma unroll
  for (int i = 0; i < WM; i++)
#pragma unroll
    for (int j = 0; j < WN; j++)
#pragma unroll
      for (int x = 0; x < 4; x++) bad |= !isfinite(acc[i][j][x]);
  if (__syncthreads_or(bad)) {
    const int64_t a0 = (int64_t)first * kBK, a1 = a0 + (int64_t)steps * kBK, nk = (int64_t)steps_a * kBK;
    for (int i = threadIdx.x; i < BM * BN; i += kThreads) {
      const size_t row = row0 + i / BN, col = col0 + i % BN;
      if (row < na && col < nb)
        atomicAdd(&S[row * nb + col], sparse_dot(ta, row, C + col, nb, a0, a1) +
                                          sparse_dot(tb, col, C + row * nb, 1, a0 - nk, a1 - nk));
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < WM; i++)
#pragma unroll
    for (int x = 0; x < 2; x++) {
      const size_t row = row0 + wm + 16 * i + 8 * x + r;
      if (row >= na) continue;
#pragma unroll
      for (int j = 0; j < WN; j++) {
        const size_t col = col0 + wn + 8 * j + 2 * q;
        if (col < nb) atomicAdd(&S[row * nb + col], acc[i][j][2 * x]);
        if (col + 1 < nb) atomicAdd(&S[row * nb + col + 1], acc[i][j][2 * x + 1]);
      }
    }
}

// one spin's string-only operator, dense, rows of ld >= n doubles
__global__ void dense_kernel(size_t n, size_t ld, Tables t, double* __restrict__ H) {
  const size_t row = blockIdx.x;
  double* h = H + row * ld;
  for (size_t j = threadIdx.x; j < ld; j += blockDim.x) h[j] = 0.0;
  __syncthreads();
  for (int64_t k = t.s_off[row] + threadIdx.x; k < t.s_off[row + 1]; k += blockDim.x) h[t.s_idx[k]] = t.s_val[k];
  for (int64_t k = t.d_off[row] + threadIdx.x; k < t.d_off[row + 1]; k += blockDim.x) h[t.d_idx[k]] = t.d_val[k];
}

template <int WM, int WN>
constexpr size_t smem_bytes() {
  return sizeof(double) * stages<WM, WN>() * (32 * WM * (kBK + 4) + kBK * (16 * WN + 4));
}

template <int WM, int WN, int V>
void launch(sbdgpu_ctx* c, const double* C, double* S) {
  dim3 grid((unsigned)((c->nb + 16 * WN - 1) / (16 * WN)), (unsigned)((c->na + 32 * WM - 1) / (32 * WM)));
  // K in shares: eight CTAs per SM, of at least four steps each (1501 x 803
  // strings, 312 tiles: 0.33 ms in one share, 0.27 in three, 0.25 in four)
  const unsigned steps = (unsigned)((c->na + kBK - 1) / kBK + (c->nb + kBK - 1) / kBK);
  grid.z = std::max(1u, std::min({(kSMs * 8u + grid.x * grid.y - 1) / (grid.x * grid.y), steps / 4, 16u}));
  allow_dynamic_smem(reinterpret_cast<const void*>(same_dense_kernel<WM, WN, V>), c->device);
  same_dense_kernel<WM, WN, V><<<grid, kThreads, smem_bytes<WM, WN>(), c->stream>>>(
      c->dense[0], c->dense_ld[0], c->dense[1], c->dense_ld[1], C, S, c->na, c->nb, view(c->tab[0]), view(c->tab[1]));
  SBD_CUDA(cudaGetLastError());
}

}  // namespace

// Whether the same-spin terms are taken as the dense product: bases with
// alpha-beta tiles, of at most 4,096 strings per spin (128 MB per operator),
// whose operators are dense enough.  The product does na nb (na + nb)
// multiply-adds at about 12 T/s, the rows kernels one per table entry and
// column at about 2.5 T/s.
bool dense_same_spin(const sbdgpu_ctx* c) {
  if (!c->tab[1].tile_grp || c->na > 4096 || c->nb > 4096) return false;
  const double na = (double)c->na, nb = (double)c->nb;
  const double entries = (double)(c->tab[0].ns + c->tab[0].nd) * nb + (double)(c->tab[1].ns + c->tab[1].nd) * na;
  return 5.0 * entries >= na * nb * (na + nb);
}

// Builds the operators where they would be used and are not there yet: by the
// FP64 sigma and the batch (an FP32 sigma has no use for them; the set-up makes
// small ones for the no-allocation sigma).  Without room for them the rows
// kernels stay.
void ensure_dense_fp64(sbdgpu_ctx* c) {
  if (c->dense[0] || c->dense_failed || c->oz.mode != 0 || !dense_same_spin(c) || !uses_tiles(c)) return;
  const size_t la = (c->na + 1) & ~size_t(1), lb = (c->nb + 1) & ~size_t(1);
  double* h = nullptr;
  try {
    h = (double*)dev_alloc(sizeof(double) * (c->na * la + c->nb * lb));
  } catch (const Error&) {
    c->dense_failed = true;
    return;
  }
  c->dense[0] = h;
  c->dense[1] = h + c->na * la;
  c->dense_ld[0] = la;
  c->dense_ld[1] = lb;
  dense_kernel<<<(unsigned)c->na, 256, 0, c->stream>>>(c->na, la, view(c->tab[0]), c->dense[0]);
  dense_kernel<<<(unsigned)c->nb, 256, 0, c->stream>>>(c->nb, lb, view(c->tab[1]), c->dense[1]);
  SBD_CUDA(cudaGetLastError());
}

void free_dense_fp64(sbdgpu_ctx* c) {
  cudaFree(c->dense[0]);
  c->dense[0] = c->dense[1] = nullptr;
  c->dense_failed = false;
}

// S += same-spin terms without the diagonal and the singles' Coulomb parts
void same_spin_dense_fp64(sbdgpu_ctx* c, const double* C, double* S) {
  // 64 x 64 tiles; 32 x 32 for the smallest bases, whose few tiles' latency
  // counts (56 x 56 strings: 4 us against 8; 495 x 495: 40 against 36)
  const bool big = ((c->na + 63) / 64) * ((c->nb + 63) / 64) >= 16;
  const bool vec = c->nb % 2 == 0 && (((uintptr_t)C | (uintptr_t)S) & 15) == 0;
  if (big) {
    if (vec) launch<2, 4, 2>(c, C, S);
    else launch<2, 4, 1>(c, C, S);
  } else {
    if (vec) launch<1, 2, 2>(c, C, S);
    else launch<1, 2, 1>(c, C, S);
  }
}

void preload_same_dense(int device) {
  allow_dynamic_smem(reinterpret_cast<const void*>(same_dense_kernel<2, 4, 2>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(same_dense_kernel<2, 4, 1>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(same_dense_kernel<1, 2, 2>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(same_dense_kernel<1, 2, 1>), device);
}

}  // namespace sbdgpu
