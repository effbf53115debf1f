// One- and two-particle RDMs (Correlation, chemistry/tpb/correlation.h:194-443)
// on the FP64 tensor pipe.
//
// In the alpha-string-major sign convention (W' = phi W) every term's sign is a
// product of one sign per spin, so that
//
//   same spin      <E_ki>, <a+_k a+_l a_j a_i> over entries (i, j) of one spin's
//                  excitation tables need only rho[i,j] = sum_k W'[i,k] W'[j,k]:
//                  a product X X^T (alpha) or X^T X (beta), then a few additions
//                  per table entry
//   opposite spin  G[ki][lj] = <E_ki E_lj> = sum over alpha entries (ia <- ja)
//                  and beta entries (ib <- jb) of s_a s_b W'[ia,ib] W'[ja,jb]:
//                  for one ja and 16 of its singles a product over ib of
//                  A[g][ib] = W'[ia_g,ib] with B[ib][rs] = s_b W'[ja, jb(ib,rs)]
//
// B is walked as k4 x n8 blocks of four neighbouring beta strings and eight
// excitation pairs; blocks without an entry are skipped (neighbouring strings
// share their pairs).  The two directions of a pair are separate accumulators.
// The columns end with the occupations (n_r of the spectators), the rows with
// ja itself (n_p for its occupied p), so that G holds every opposite-spin
// element.  Of the alpha pairs only k > i is taken: <E_ki E_lj> = <E_ik E_jl>.
//
// Per pair of determinants this is one multiply-add on the tensor pipe where
// the scalar kernels (rdm.cu) do one warp-wide gather of two shared-memory
// values: 1M determinants, norb 20, 8.2 -> 1.3 ms of kernels, 11.4 -> 4.2-4.9 ms
// a call.
#include <algorithm>

#include "device.cuh"
#include "internal.cuh"

namespace sbdgpu {

namespace {

constexpr int kThreads = 128;   // products
constexpr int kBK = 16;
constexpr int kStages = 4;
constexpr int kAbThreads = 256;  // opposite spins
constexpr int kWarpTiles = 4;    // n8 tiles per warp
constexpr int kCtaTiles = kWarpTiles * kAbThreads / 32;

__device__ __forceinline__ void copy8(double* dst, const double* src, bool on) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = on ? 8 : 0;  // the rest is zero-filled
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// rho[i - i0][j] for rows i0 .. i0 + rows of the n x n matrix X X^T (TRANS
// false: X row-major n x depth) or X^T X (TRANS: X row-major depth x n).
// CTA tiles of 64 x 64, each warp 32 x 32.
template <bool TRANS>
__global__ void __launch_bounds__(kThreads) rho_kernel(const double* __restrict__ X, size_t n, size_t depth, size_t i0,
                                                      size_t rows, double* __restrict__ rho) {
  // staged as [64][kBK + 4] (rows of X) or [kBK][64 + 4]: conflict-free fragments
  constexpr int P = TRANS ? 68 : kBK + 4, TILE = TRANS ? kBK * 68 : 64 * (kBK + 4);
  extern __shared__ __align__(16) double smem_d[];
  const size_t row0 = i0 + (size_t)blockIdx.y * 64, col0 = (size_t)blockIdx.x * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, q = lane & 3;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int steps = (int)((depth + kBK - 1) / kBK);
  const auto load = [&](double* dst, size_t first, size_t k0) {
    for (int i = threadIdx.x; i < 64 * kBK; i += kThreads) {
      if constexpr (TRANS) {
        const int k = i >> 6, m = i & 63;
        const bool on = k0 + k < depth && first + m < n;
        copy8(dst + k * P + m, on ? X + (k0 + k) * n + first + m : X, on);
      } else {
        const int m = i / kBK, k = i % kBK;
        const bool on = k0 + k < depth && first + m < n;
        copy8(dst + m * P + k, on ? X + (first + m) * depth + k0 + k : X, on);
      }
    }
  };
  const auto fetch = [&](int s) {
    if (s < steps) {
      double* t = smem_d + (size_t)(s % kStages) * 2 * TILE;
      load(t, row0, (size_t)s * kBK);
      load(t + TILE, col0, (size_t)s * kBK);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[2][4][4] = {};
  for (int s = 0; s < kStages - 1; s++) fetch(s);
  for (int s = 0; s < steps; s++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    fetch(s + kStages - 1);
    const double* a = smem_d + (size_t)(s % kStages) * 2 * TILE;
    const double* b = a + TILE;
    const auto at = [&](const double* t, int m, int k) { return TRANS ? t[k * P + m] : t[m * P + k]; };
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double fa[2][2], fb[4];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        fa[i][0] = at(a, wm + 16 * i + r, kk + q);
        fa[i][1] = at(a, wm + 16 * i + 8 + r, kk + q);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) fb[j] = at(b, wn + 8 * j + r, kk + q);
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) mma16(acc[i][j], fa[i][0], fa[i][1], fb[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const size_t row = row0 + wm + 16 * i + 8 * (x >> 1) + r, col = col0 + wn + 8 * j + 2 * q + (x & 1);
        if (row < i0 + rows && row < n && col < n) rho[(row - i0) * n + col] = acc[i][j][x];
      }
}

__device__ __forceinline__ int low_bit(uint64_t x) { return __ffsll((long long)x) - 1; }
__device__ __forceinline__ bool odd_between(uint64_t s, int p, int q) {
  const int lo = min(p, q), hi = max(p, q);
  const uint64_t mask = hi - lo < 2 ? 0ull : (((1ull << hi) - 1ull) & ~((2ull << lo) - 1ull));
  return __popcll(s & mask) & 1;
}

// The same-spin elements of spin S from rho rows i0 ..: one block per bra
// string, one thread per table entry; the diagonal of rho goes to dia.
__global__ void __launch_bounds__(128) same_spin_kernel(int S, const double* __restrict__ rho, size_t n, size_t i0,
                                                       const uint64_t* __restrict__ str, int L,
                                                       const int64_t* __restrict__ s_off,
                                                       const int32_t* __restrict__ s_idx,
                                                       const uint32_t* __restrict__ s_info,
                                                       const int64_t* __restrict__ d_off,
                                                       const int32_t* __restrict__ d_idx, double* __restrict__ one,
                                                       double* __restrict__ two, double* __restrict__ dia) {
  const size_t i = i0 + blockIdx.x;
  const double* row = rho + (size_t)blockIdx.x * n;
  const size_t L1 = L, L2 = L1 * L1, L3 = L2 * L1;
  double* t = two + (size_t)(3 * S) * L2 * L2;
  // <c1+ c2+ a2 a1> at a1 + L a2 + L^2 c1 + L^3 c2
  const auto add = [&](int c1, int c2, int a2, int a1, double v) {
    atomicAdd(&t[a1 + L1 * a2 + L2 * c1 + L3 * c2], v);
  };
  if (threadIdx.x == 0) dia[i] = row[i];
  const int64_t s0 = s_off[i], ns = s_off[i + 1] - s0, d0 = d_off[i], nd = d_off[i + 1] - d0;
  for (int64_t k = threadIdx.x; k < ns + nd; k += blockDim.x) {
    if (k < ns) {
      const int32_t j = s_idx[s0 + k];
      const uint32_t info = s_info[s0 + k];
      const int p = info & 63, q = (info >> 6) & 63;  // created, annihilated
      const double v = info & 0x80000000u ? -row[j] : row[j];
      if (v == 0.0) continue;
      atomicAdd(&one[S * L2 + p + L1 * q], v);
      // Spectators of this spin.  The created orbital's own terms cancel: they are
      // added, as the reference adds them, only where their difference is a NaN.
      for (uint64_t o = isfinite(v) ? str[i] & str[j] : str[i]; o; o &= o - 1) {
        const int r = low_bit(o);
        add(p, r, r, q, v);
        add(r, p, q, r, v);
        add(p, r, q, r, -v);
        add(r, p, r, q, -v);
      }
    } else {
      const int32_t j = d_idx[d0 + (k - ns)];
      const uint64_t si = str[i], sj = str[j], c = si & ~sj, d = sj & ~si;
      const int p1 = low_bit(c), p2 = low_bit(c & (c - 1)), q1 = low_bit(d), q2 = low_bit(d & (d - 1));
      bool neg = odd_between(sj, q1, p1) ^ odd_between(sj, q2, p2);
      if (p1 > q2 || p2 < q1) neg = !neg;
      const double v = neg ? -row[j] : row[j];
      if (v == 0.0) continue;
      add(p1, p2, q2, q1, v);
      add(p2, p1, q1, q2, v);
      add(p1, p2, q1, q2, -v);
      add(p2, p1, q2, q1, -v);
    }
  }
}

// Beta entries by (four strings, eight columns): ket | forward << 30 | sign <<
// 31 at lane 4 column + string, an empty slot's ket being nb; flags: bit 0 a
// forward entry (the bra holds the pair's higher orbital; every occupation),
// bit 1 a backward one.  Columns: off-diagonal pairs, then the L occupations.
__global__ void __launch_bounds__(256) entries_kernel(size_t nb, int L, int ntile, const uint64_t* __restrict__ bstr,
                                                     const int64_t* __restrict__ s_off,
                                                     const int32_t* __restrict__ s_idx,
                                                     const uint32_t* __restrict__ s_info, uint32_t* __restrict__ ent,
                                                     uint32_t* __restrict__ flags) {
  extern __shared__ uint32_t fl[];  // [ntile]
  const size_t quad = blockIdx.x;
  uint32_t* e = ent + quad * ntile * 32;
  const int npair = L * (L - 1) / 2;
  for (int i = threadIdx.x; i < ntile * 32; i += blockDim.x) e[i] = (uint32_t)nb;
  for (int i = threadIdx.x; i < ntile; i += blockDim.x) fl[i] = 0;
  __syncthreads();
  const auto put = [&](int col, int k, uint32_t word) {
    e[(size_t)(col >> 3) * 32 + (col & 7) * 4 + k] = word;
    atomicOr(&fl[col >> 3], word & 0x40000000u ? 1u : 2u);
  };
  for (int k = 0; k < 4; k++) {
    const size_t ib = quad * 4 + k;
    if (ib >= nb) break;
    for (int64_t x = s_off[ib] + threadIdx.x; x < s_off[ib + 1]; x += blockDim.x) {
      const uint32_t info = s_info[x];
      const int p = info & 63, q = (info >> 6) & 63;
      put(od_pair(p, q), k, (uint32_t)s_idx[x] | (p > q ? 0x40000000u : 0u) | (info & 0x80000000u));
    }
    for (int r = threadIdx.x; r < L; r += blockDim.x)
      if ((bstr[ib] >> r) & 1ull) put(npair + r, k, (uint32_t)ib | 0x40000000u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ntile; i += blockDim.x) flags[quad * ntile + i] = fl[i];
}

// G[row][direction][column] += the products of one ja, 16 of its rows (alpha
// singles that create above what they annihilate, then ja itself) and 32
// column tiles; W' in Wp.  kSmem: the row of ja in shared memory.
template <bool kSmem>
__global__ void __launch_bounds__(kAbThreads) opposite_spin_kernel(
    const double* __restrict__ Wp, size_t nb, const uint64_t* __restrict__ astr, int L, int ntile,
    const int64_t* __restrict__ a_off, const int32_t* __restrict__ a_idx, const uint32_t* __restrict__ a_info,
    const uint32_t* __restrict__ ent, const uint32_t* __restrict__ flags, double* __restrict__ G) {
  extern __shared__ __align__(16) double crow[];  // [nb + 1], the last one zero
  __shared__ int tgt[16], gpair[16];
  __shared__ uint32_t gneg[16];
  __shared__ int nrow;
  const size_t ja = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, q = lane & 3;
  const int first = (int)blockIdx.y * 16;
  if (threadIdx.x < 16) tgt[threadIdx.x] = -1;
  __syncthreads();
  if (warp == 0) {
    int rank = 0;
    for (int64_t k0 = a_off[ja]; k0 < a_off[ja + 1]; k0 += 32) {
      const int64_t k = k0 + lane;
      const bool in = k < a_off[ja + 1];
      const uint32_t info = in ? a_info[k] : 0u;
      // the table's bra is ja: its created orbital is what ia <- ja annihilates
      const int ann = info & 63, cre = (info >> 6) & 63;
      const unsigned up = __ballot_sync(0xffffffffu, in && cre > ann);
      const int at = rank + __popc(up & ((1u << lane) - 1u)) - first;
      if (in && cre > ann && at >= 0 && at < 16) {
        tgt[at] = a_idx[k];
        gpair[at] = od_pair(cre, ann);
        gneg[at] = info & 0x80000000u;
      }
      rank += __popc(up);
    }
    if (lane == 0) {
      const int at = rank - first;  // ja itself comes last
      if (at >= 0 && at < 16) {
        tgt[at] = (int)ja;
        gpair[at] = -1;
        gneg[at] = 0;
      }
      nrow = at + 1;
    }
  }
  __syncthreads();
  if (nrow <= 0) return;
  if (kSmem) {
    for (size_t i = threadIdx.x; i <= nb; i += kAbThreads) crow[i] = i < nb ? Wp[ja * nb + i] : 0.0;
    __syncthreads();
  }
  const double* wrow = Wp + ja * nb;
  const double* ra = tgt[r] >= 0 ? Wp + (size_t)tgt[r] * nb : nullptr;
  const double* rb = tgt[r + 8] >= 0 ? Wp + (size_t)tgt[r + 8] * nb : nullptr;
  const int t0 = (int)blockIdx.z * kCtaTiles + warp * kWarpTiles;
  const int nt = min(kWarpTiles, ntile - t0);
  const size_t quads = (nb + 3) / 4;
  double acc[kWarpTiles][2][4] = {};
  double a0 = 0.0, a1 = 0.0;
  uint32_t e[kWarpTiles], f[kWarpTiles];
  const auto fetch = [&](size_t quad) {  // the operands of one quad, a step ahead
    const size_t ib = quad * 4 + q;
    a0 = ra && ib < nb ? __ldg(&ra[ib]) : 0.0;
    a1 = rb && ib < nb ? __ldg(&rb[ib]) : 0.0;
#pragma unroll
    for (int i = 0; i < kWarpTiles; i++) {
      f[i] = i < nt ? __ldg(&flags[quad * ntile + t0 + i]) : 0u;
      e[i] = i < nt ? __ldg(&ent[(quad * ntile + t0 + i) * 32 + lane]) : (uint32_t)nb;
    }
  };
  if (nt > 0) {
    fetch(0);
    for (size_t quad = 0; quad < quads; quad++) {
      const double x0 = a0, x1 = a1;
      uint32_t ec[kWarpTiles], fc[kWarpTiles];
#pragma unroll
      for (int i = 0; i < kWarpTiles; i++) {
        ec[i] = e[i];
        fc[i] = f[i];
      }
      if (quad + 1 < quads) fetch(quad + 1);
#pragma unroll
      for (int i = 0; i < kWarpTiles; i++) {
        if (!fc[i]) continue;  // the same in every lane
        const uint32_t ket = ec[i] & 0xFFFFu;
        double w = kSmem ? crow[ket] : ket < nb ? __ldg(&wrow[ket]) : 0.0;
        if (ec[i] & 0x80000000u) w = -w;
        const bool fwd = ec[i] & 0x40000000u;
        if (fc[i] & 1u) mma16(acc[i][0], x0, x1, fwd ? w : 0.0);
        if (fc[i] & 2u) mma16(acc[i][1], x0, x1, fwd ? 0.0 : w);
      }
    }
  }
  const size_t ncol = (size_t)ntile * 8;
  const int npair = L * (L - 1) / 2;
  const auto add = [&](int g, int d, int t, int col, double v) {
    if (v == 0.0) return;
    const size_t at = d * ncol + (size_t)t * 8 + col;
    if (gpair[g] >= 0) {
      atomicAdd(&G[(size_t)gpair[g] * 2 * ncol + at], v);
    } else {
      for (uint64_t o = astr[ja]; o; o &= o - 1) atomicAdd(&G[(size_t)(npair + low_bit(o)) * 2 * ncol + at], v);
    }
  };
  // A NaN or an infinity times the zero of an empty slot reaches columns that no
  // entry of its beta string has: the warp's elements entry by entry instead.
  bool bad = false;
#pragma unroll
  for (int i = 0; i < kWarpTiles; i++)
#pragma unroll
    for (int d = 0; d < 2; d++)
#pragma unroll
      for (int x = 0; x < 4; x++) bad |= !isfinite(acc[i][d][x]);
  if (__any_sync(0xffffffffu, bad)) {
    for (int x = lane; x < 16 * nt * 8; x += 32) {
      const int g = x & 15, t = t0 + (x >> 7), col = (x >> 4) & 7;
      if (tgt[g] < 0) continue;
      const double* arow = Wp + (size_t)tgt[g] * nb;
      double fwd = 0.0, back = 0.0;
      for (size_t ib = 0; ib < nb; ib++) {
        const uint32_t w = __ldg(&ent[((ib >> 2) * ntile + t) * 32 + col * 4 + (ib & 3)]);
        if ((w & 0xFFFFu) == (uint32_t)nb) continue;
        const double y = arow[ib] * ((w ^ gneg[g]) & 0x80000000u ? -wrow[w & 0xFFFFu] : wrow[w & 0xFFFFu]);
        if (w & 0x40000000u)
          fwd += y;
        else
          back += y;
      }
      add(g, 0, t, col, fwd);
      add(g, 1, t, col, back);
    }
    return;
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int g = r + 8 * h;
    if (tgt[g] < 0) continue;
    const double s = gneg[g] ? -1.0 : 1.0;
#pragma unroll
    for (int i = 0; i < kWarpTiles; i++) {
      if (i >= nt) break;
#pragma unroll
      for (int d = 0; d < 2; d++)
#pragma unroll
        for (int u = 0; u < 2; u++) add(g, d, t0 + i, 2 * q + u, s * acc[i][d][2 * h + u]);
    }
  }
}

// G into the two opposite-spin blocks of the two-particle array.  A double
// excitation whose lower created and lower annihilated spin orbitals differ in
// spin goes to the other block, as TwoDiffCorrelation (correlation.h:91-130)
// puts it.
__global__ void opposite_spin_place_kernel(const double* __restrict__ G, int L, int ntile, double* __restrict__ two) {
  const int P = L * (L + 1) / 2, npair = L * (L - 1) / 2;
  const size_t ncol = (size_t)ntile * 8, L1 = L, L2 = L1 * L1, L4 = L2 * L2;
  const auto orbitals = [&](int x, int& hi, int& lo) {
    if (x >= npair) {
      hi = lo = x - npair;
      return;
    }
    hi = od_larger(x);
    lo = x - hi * (hi - 1) / 2;
  };
  // <E_ki (alpha) E_lj (beta)>
  const auto put = [&](size_t k, size_t i, size_t l, size_t j, double v) {
    const bool other = k != i && l != j && (k <= l) != (i <= j);
    atomicAdd(&two[(other ? 1 : 2) * L4 + i + L1 * j + L2 * k + L2 * L1 * l], v);  // two quadruples may share an entry
    atomicAdd(&two[(other ? 2 : 1) * L4 + j + L1 * i + L2 * l + L2 * L1 * k], v);
  };
  for (size_t x = (size_t)blockIdx.x * blockDim.x + threadIdx.x; x < (size_t)P * P * 2;
       x += (size_t)gridDim.x * blockDim.x) {
    const int d = (int)(x % 2), b = (int)(x / 2 % P), a = (int)(x / 2 / P);
    if (d == 1 && b >= npair) continue;
    const double v = G[(size_t)a * 2 * ncol + d * ncol + b];
    if (v == 0.0) continue;
    int k, i, hi, lo;
    orbitals(a, k, i);
    orbitals(b, hi, lo);
    const int l = d == 0 ? hi : lo, j = d == 0 ? lo : hi;
    put(k, i, l, j, v);
    if (k != i) put(i, k, j, l, v);
  }
}

}  // namespace

// one [2][L^2] and two [4][L^4] += every element of W' W' but the same-spin
// diagonal ones; dia [na + nb]: the strings' weights.  False, with nothing done,
// where device memory has no room for its tables.
bool rdm_products(sbdgpu_ctx* c, const double* Wp, double* one, double* two, double* dia) {
  const int L = c->L, P = c->P, ntile = (P + 7) / 8;
  const size_t na = c->na, nb = c->nb, quads = (nb + 3) / 4, ncol = (size_t)ntile * 8;
  cudaStream_t st = c->stream;
  // rho in row panels of at most 1 GiB
  const size_t nmax = std::max(na, nb);
  const size_t panel = std::max<size_t>(64, (size_t(1) << 27) / nmax / 64 * 64);
  double *rho = nullptr, *G = nullptr;
  uint32_t *ent = nullptr, *flags = nullptr;
  Arena arena(st);
  arena.add(&rho, std::max(std::min(panel, na) * na, std::min(panel, nb) * nb));
  arena.add(&G, (size_t)P * 2 * ncol);
  arena.add(&ent, quads * ntile * 32);
  arena.add(&flags, quads * ntile);
  try {
    arena.commit();
  } catch (const Error&) {
    return false;
  }
  SBD_CUDA(cudaMemsetAsync(G, 0, sizeof(double) * P * 2 * ncol, st));
  const SpinTables& ta = c->tab[0];
  const SpinTables& tb = c->tab[1];
  entries_kernel<<<(unsigned)quads, 256, sizeof(uint32_t) * ntile, st>>>(nb, L, ntile, c->bstr, tb.s_off, tb.s_idx,
                                                                         tb.s_info, ent, flags);
  SBD_CUDA(cudaGetLastError());
  const dim3 grid((unsigned)na, (unsigned)((ta.max_s + 1 + 15) / 16), (unsigned)((ntile + kCtaTiles - 1) / kCtaTiles));
  int optin = 0;
  SBD_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const size_t row = sizeof(double) * (nb + 1);
  if (row + 1024 <= (size_t)optin) {
    allow_dynamic_smem(reinterpret_cast<const void*>(opposite_spin_kernel<true>), c->device);
    opposite_spin_kernel<true><<<grid, kAbThreads, row, st>>>(Wp, nb, c->astr, L, ntile, ta.s_off, ta.s_idx, ta.s_info,
                                                             ent, flags, G);
  } else {
    opposite_spin_kernel<false><<<grid, kAbThreads, 0, st>>>(Wp, nb, c->astr, L, ntile, ta.s_off, ta.s_idx, ta.s_info,
                                                            ent, flags, G);
  }
  SBD_CUDA(cudaGetLastError());
  opposite_spin_place_kernel<<<kSMs * 4, 256, 0, st>>>(G, L, ntile, two);
  SBD_CUDA(cudaGetLastError());
  for (int S = 0; S < 2; S++) {
    const SpinTables& t = S == 0 ? ta : tb;
    const size_t n = S == 0 ? na : nb, depth = S == 0 ? nb : na;
    for (size_t i0 = 0; i0 < n; i0 += panel) {
      const size_t rows = std::min(panel, n - i0);
      const dim3 g((unsigned)((n + 63) / 64), (unsigned)((rows + 63) / 64));
      if (S == 0) {
        constexpr size_t smem = sizeof(double) * kStages * 2 * 64 * (kBK + 4);
        allow_dynamic_smem(reinterpret_cast<const void*>(rho_kernel<false>), c->device);
        rho_kernel<false><<<g, kThreads, smem, st>>>(Wp, n, depth, i0, rows, rho);
      } else {
        constexpr size_t smem = sizeof(double) * kStages * 2 * kBK * 68;
        allow_dynamic_smem(reinterpret_cast<const void*>(rho_kernel<true>), c->device);
        rho_kernel<true><<<g, kThreads, smem, st>>>(Wp, n, depth, i0, rows, rho);
      }
      SBD_CUDA(cudaGetLastError());
      same_spin_kernel<<<(unsigned)rows, 128, 0, st>>>(S, rho, n, i0, S == 0 ? c->astr : c->bstr, L, t.s_off, t.s_idx,
                                                       t.s_info, t.d_off, t.d_idx, one, two, dia + (S ? na : 0));
      SBD_CUDA(cudaGetLastError());
    }
  }
  SBD_CUDA(cudaStreamSynchronize(st));
  return true;
}

}  // namespace sbdgpu
