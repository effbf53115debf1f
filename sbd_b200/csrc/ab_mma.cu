// The alpha-beta term of sigma on the FP64 tensor pipe (the reference's task
// type 0, chemistry/tpb/mult.h:567-611):
//
//   sigma[ia,ib] += sum_{ja in S(ia)} sum_{jb in S(ib)} s_a s_b (pq|rs) C[ja,jb]
//
// For one source string ja and the singles g = 1..M of one CTA this is a
// product per beta string, y_g(ib) = sum_rs (pq_g|rs) x_rs(ib) with
// x_rs(ib) = s_b C[ja, jb(ib, rs)], sparse in rs.  Neighbouring beta strings
// (ascending strings share their high orbitals) have most of their excitation
// pairs rs in common, so eight of them are taken as the N dimension of an FP64
// mma.m16n8k4 whose K runs over the union of their pairs; strings without a
// pair contribute a zero.  At norb 36, 8 electrons and 12,000 strings 63 % of
// the slots are filled, at norb 26 / 6 / 4,000 53 %, and an operand of the
// integrals then feeds 8 or 16 beta strings instead of one: a gather of one
// integral per multiply-add is bound by the shared-memory pipe at a quarter of
// the FP64 rate.
//
// Tiles (built once per context): beta strings in groups of 16, two n8 tiles
// each.  The pairs both tiles use come first (one load of the integrals feeds
// both), then those of the first tile alone, then those of the second, each
// section in whole k4 steps.  Within a section the pairs are dealt to the
// steps so that the four pairs of a step differ modulo 4 while the classes
// last: the integral rows are turned by that class and the four rows then lie
// in different banks.  One 32-bit entry per slot, in the order of the B
// fragment (lane = 4 n + k); an empty slot points at a zero behind the row of
// C.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "internal.cuh"

namespace sbdgpu {

namespace {

constexpr int kMmaThreads = 1024;
constexpr int kMaxWords = 63;  // bitmap words of the off-diagonal pairs: 64 * 63 / 2 = 2016

__device__ __forceinline__ int od_pair(uint32_t info) {  // off-diagonal pair index of a single
  const int p = info & 63, q = (info >> 6) & 63;
  const int hi = max(p, q), lo = min(p, q);
  return hi * (hi - 1) / 2 + lo;
}

// The folded pair (diagonal ones included) of off-diagonal pair o: the larger
// orbital hi has hi (hi - 1) / 2 <= o < hi (hi + 1) / 2, and hi diagonal
// pairs come before.
__device__ __forceinline__ int folded_pair(int o) {
  int hi = (int)((1.0f + sqrtf(8.0f * (float)o + 1.0f)) * 0.5f);
  hi += hi * (hi + 1) / 2 <= o;
  hi -= hi * (hi - 1) / 2 > o;
  return o + hi;
}

// Bitmaps of the pairs used by the two tiles of a group, then the words of one
// section (0: both tiles, 1: the first alone, 2: the second alone).
__device__ __forceinline__ void tile_bitmaps(uint32_t (*bm)[kMaxWords + 1], int words, int n, int g,
                                             const int64_t* __restrict__ s_off, const uint32_t* __restrict__ s_info) {
  const int lane = threadIdx.x;
  for (int w = lane; w < words; w += 32) bm[0][w] = bm[1][w] = 0;
  __syncwarp();
  for (int t = 0; t < 2; t++) {
    const int i0 = min(g * 16 + t * 8, n), i1 = min(i0 + 8, n);
    for (int64_t k = s_off[i0] + lane; k < s_off[i1]; k += 32) {
      const int o = od_pair(s_info[k]);
      atomicOr(&bm[t][o >> 5], 1u << (o & 31));
    }
  }
  __syncwarp();
}
__device__ __forceinline__ uint32_t section_word(const uint32_t (*bm)[kMaxWords + 1], int sec, int w) {
  const uint32_t a = bm[0][w], b = bm[1][w];
  return sec == 0 ? (a & b) : sec == 1 ? (a & ~b) : (b & ~a);
}

// k4 steps of each group: {-, both tiles, the first alone, the second alone}
__global__ void __launch_bounds__(32) tile_count_kernel(int n, int words, const int64_t* __restrict__ s_off,
                                                       const uint32_t* __restrict__ s_info, int4* __restrict__ grp) {
  __shared__ uint32_t bm[2][kMaxWords + 1];
  const int g = blockIdx.x, lane = threadIdx.x;
  tile_bitmaps(bm, words, n, g, s_off, s_info);
  int c[3] = {0, 0, 0};
  for (int w = lane; w < words; w += 32)
    for (int s = 0; s < 3; s++) c[s] += __popc(section_word(bm, s, w));
  for (int o = 16; o; o >>= 1)
    for (int s = 0; s < 3; s++) c[s] += __shfl_xor_sync(0xffffffffu, c[s], o);
  if (lane == 0) grp[g] = make_int4(0, (c[0] + 3) / 4, (c[1] + 3) / 4, (c[2] + 3) / 4);
}

__global__ void __launch_bounds__(32) tile_fill_kernel(int n, int words, const int64_t* __restrict__ s_off,
                                                      const int32_t* __restrict__ s_idx,
                                                      const uint32_t* __restrict__ s_info,
                                                      const int4* __restrict__ grp, uint32_t* __restrict__ ent) {
  __shared__ uint32_t bm[2][kMaxWords + 1];
  __shared__ int pre[3][4][kMaxWords + 1];  // pairs of a section and class in earlier words
  __shared__ int cnt[3][4];
  const int g = blockIdx.x, lane = threadIdx.x;
  tile_bitmaps(bm, words, n, g, s_off, s_info);
  if (lane < 12) {
    const int s = lane >> 2, c = lane & 3;
    int acc = 0;
    for (int w = 0; w < words; w++) {
      pre[s][c][w] = acc;
      acc += __popc(section_word(bm, s, w) & (0x11111111u << c));
    }
    cnt[s][c] = acc;
  }
  __syncwarp();
  const int4 d = grp[g];
  uint32_t* base = ent + (size_t)d.x * 32;
  const uint32_t zero = (uint32_t)n << 3;  // the zero behind the row of C
  const auto first_word = [](uint32_t ket, int o, bool neg) {
    return (neg ? 1u : 0u) | ket << 3 | (uint32_t)(o << 2 | (o & 3)) << 19;
  };
  const auto second_word = [](uint32_t ket, bool neg) { return ket << 3 | (neg ? 0x80000000u : 0u); };
  const int64_t total = 32ll * (2 * d.y + d.z + d.w);
  for (int64_t k = lane; k < total; k += 32) base[k] = zero;
  __syncwarp();
  // a pair's place in its section: by (rank in its class, class)
  auto place = [&](int o, int s) {
    const int c = o & 3, w = o >> 5;
    const uint32_t below = section_word(bm, s, w) & (0x11111111u << c) & ((1u << (o & 31)) - 1u);
    const int r = pre[s][c][w] + __popc(below);
    int at = 0;
    for (int x = 0; x < 4; x++) at += min(cnt[s][x], r) + (x < c && cnt[s][x] > r);
    return at;
  };
  // entry of beta string `nn` (0..7) of tile t at place `at` of section s
  auto slot = [&](int s, int at, int nn, int t) {
    const int step = at >> 2, lane_of = nn * 4 + (at & 3);
    if (s == 0) return ((size_t)step * 32 + lane_of) * 2 + t;
    return (size_t)(2 * d.y + (s == 2 ? d.z : 0) + step) * 32 + lane_of;
  };
  // every slot of a pair names the pair (the A operand of the whole column)
  for (int o = lane; o < words * 32; o += 32)
    for (int s = 0; s < 3; s++)
      if ((section_word(bm, s, o >> 5) >> (o & 31)) & 1u) {
        const int at = place(o, s);
        for (int nn = 0; nn < 8; nn++) base[slot(s, at, nn, 0)] = first_word((uint32_t)n, o, false);
      }
  __syncwarp();
  for (int t = 0; t < 2; t++)
    for (int nn = 0; nn < 8; nn++) {
      const int i = g * 16 + t * 8 + nn;
      if (i >= n) break;
      for (int64_t k = s_off[i] + lane; k < s_off[i + 1]; k += 32) {
        const uint32_t info = s_info[k];
        const int o = od_pair(info);
        const bool other = (bm[1 - t][o >> 5] >> (o & 31)) & 1u;
        const int s = other ? 0 : 1 + t;
        const uint32_t ket = (uint32_t)s_idx[k];
        const bool neg = info >> 31;
        base[slot(s, place(o, s), nn, t)] = s == 0 && t == 1 ? second_word(ket, neg) : first_word(ket, o, neg);
      }
    }
}

// D (16 x 8) += A (16 x 4) B (4 x 8), FP64
__device__ __forceinline__ void mma16(double (&d)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5},{%6},{%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b));
}
// D (8 x 8) += A (8 x 4) B (4 x 8), FP64
__device__ __forceinline__ void mma8(double (&d)[4], double a0, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a0), "d"(b));
}

// FP32 vectors: the row of C is converted as it is staged, products and sums
// stay FP64, a row's sum is rounded once before it is added.
//
// What bounds it: the shared-memory pipe (16M determinants: 86 % of its
// wavefronts, the FP64 tensor pipe 68 % busy).  Alpha-beta term, gather kernel
// -> tiles: 144M determinants 198 -> 89 ms, 16M 11.2 -> 4.0 ms, 1501 x 803
// strings 0.85 -> 0.34 ms, 495 x 495 0.10 -> 0.052 ms; the tensor pipe's floor
// of the filled tiles is 54 / 2.8 ms at the first two.  24 and 32 alpha
// singles per CTA (fewer loads of C per product) and entries fetched a batch
// ahead were no faster: fewer warps fit, and the loads were not what waited.
//
// Entries.  Word of a tile alone, and of the first of two: sign | ket << 3 |
// row << 19 with row = pair << 2 | (pair & 3); word of the second tile where
// both share the pair: ket << 3 | sign << 31.  The integral arrays hold 16 (or 8) doubles per pair in
// 32-byte chunks whose order is turned by the pair's class modulo 4, so the
// byte offset of a lane's operands is the row field, shifted and masked, xor a
// constant of the lane.
template <int W>
__device__ __forceinline__ uint32_t lane_bits(int r) {
  if constexpr (W == 16) return (((uint32_t)r >> 1) << 5) | (((uint32_t)r & 1u) << 4);
  return (((uint32_t)r >> 2) << 5) | (((uint32_t)r & 3u) << 3);
}
template <int W>
__device__ __forceinline__ uint32_t row_offset(uint32_t e, uint32_t lbits) {
  if constexpr (W == 16) return ((e >> 14) & 0x3FFE0u) ^ lbits;
  return ((e >> 15) & 0x1FFE0u) ^ lbits;
}
template <int W>
__device__ __forceinline__ uint32_t store_offset(int o, int place) {  // where `place` of a pair's row lies
  if constexpr (W == 16) return ((uint32_t)o << 7) + (((uint32_t)place >> 2 ^ ((uint32_t)o & 3u)) << 5) + ((place & 3) << 3);
  return ((uint32_t)o << 6) + (((uint32_t)place >> 2 ^ (((uint32_t)o >> 1) & 1u)) << 5) + ((place & 3) << 3);
}

__device__ __forceinline__ double c_value(const unsigned char* crow, uint32_t e, uint32_t sign) {
  const double x = *reinterpret_cast<const double*>(crow + (e & 0x7FFF8u));
  return __hiloint2double(__double2hiint(x) ^ (int)sign, __double2loint(x));
}

// acc[t] += the CTA's integrals of a step's four pairs x B of tile t: two m8
// blocks of alpha singles (M = 16: their rows interleaved, so that one 16-byte
// load feeds an m16 product) or, BLOCKS = 1, the first alone
template <int M, int BLOCKS, int NT>
__device__ __forceinline__ void products(const unsigned char* vsub, uint32_t lbits, uint32_t e, const double (&b)[NT],
                                         double (*const (&acc)[NT])[4]) {
  const unsigned char* va = vsub + row_offset<M>(e, lbits);
  if constexpr (BLOCKS == 2) {
    const double2 a = *reinterpret_cast<const double2*>(va);
#pragma unroll
    for (int t = 0; t < NT; t++) mma16(*acc[t], a.x, a.y, b[t]);
  } else {
    const double a = *reinterpret_cast<const double*>(va);
#pragma unroll
    for (int t = 0; t < NT; t++) mma8(*acc[t], a, b[t]);
  }
}

template <typename T>
struct MmaArgs {
  const T* C;
  T* S;
  size_t na, nb, ia0;
  int P, npair;
  const double* vf;
  const int64_t* a_off;
  const int32_t* a_idx;
  const uint32_t* a_info;
  const int4* grp;
  const uint32_t* ent;
  int ngroup;
  int bulk;  // rows of S start on 16 bytes wherever a group of beta strings does
  const double* Ja;  // [P][na]: the beta singles' Coulomb part as well (null: not)
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// dst += staged values, by the copy engine (16-byte aligned addresses, bytes a
// multiple of 16)
__device__ __forceinline__ void bulk_add(double* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(dst), "r"(src),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void bulk_add(float* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(src),
               "r"(bytes)
               : "memory");
}

// A section of n steps (uint2 entries: both tiles, uint32_t: one), the entries
// of four steps in flight.
template <typename E, class F>
__device__ __forceinline__ void section(const E* __restrict__ p, int n, F&& step) {
  int s = 0;
  for (; s + 4 <= n; s += 4, p += 128) {
    E e[4];
#pragma unroll
    for (int u = 0; u < 4; u++) e[u] = __ldg(&p[u * 32]);
#pragma unroll
    for (int u = 0; u < 4; u++) step(e[u]);
  }
  if (s < n) {
    E e[3];
#pragma unroll
    for (int u = 0; u < 3; u++)
      if (s + u < n) e[u] = __ldg(&p[u * 32]);
#pragma unroll
    for (int u = 0; u < 3; u++)
      if (s + u < n) step(e[u]);
  }
}

// The groups of 16 beta strings of one warp.  stage: the warp's [8 SB][16]
// results of SB blocks of alpha singles, whose rows are added to sigma as whole 128-byte lines: by the
// copy engine where they start on 16 bytes, else by coalesced atomics.  (Added
// straight from the accumulators' layout, 8 rows x 2 columns per lane, the
// atomics took 29 % of the shared-memory pipe's wavefronts.)
template <typename T, int M, int BLOCKS, int SB>
__device__ __forceinline__ void tiles(const MmaArgs<T>& a, const unsigned char* vsub, const unsigned char* crow,
                                      T* stage, const int* tgt, const uint32_t* neg) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int r = lane >> 2, q = lane & 3;
  const uint32_t lbits = lane_bits<M>(r);
  for (int g = warp; g < a.ngroup; g += nwarp) {
    const int4 d = __ldg(&a.grp[g]);
    const uint32_t* p = a.ent + (size_t)d.x * 32;
    double acc0[4] = {0.0, 0.0, 0.0, 0.0}, acc1[4] = {0.0, 0.0, 0.0, 0.0};
    section(reinterpret_cast<const uint2*>(p) + lane, d.y, [&](uint2 x) {
      const double b[2] = {c_value(crow, x.x, x.x << 31), c_value(crow, x.y, x.y & 0x80000000u)};
      double(*const both[2])[4] = {&acc0, &acc1};
      products<M, BLOCKS, 2>(vsub, lbits, x.x, b, both);
    });
    const auto alone = [&](const uint32_t* words, int n, double(&acc)[4]) {
      section(words, n, [&](uint32_t x) {
        const double b[1] = {c_value(crow, x, x << 31)};
        double(*const one[1])[4] = {&acc};
        products<M, BLOCKS, 1>(vsub, lbits, x, b, one);
      });
    };
    alone(p + (size_t)64 * d.y + lane, d.z, acc0);
    alone(p + (size_t)64 * d.y + (size_t)32 * d.z + lane, d.w, acc1);
    const size_t ib0 = (size_t)g * 16;
#pragma unroll
    for (int b0 = 0; b0 < BLOCKS; b0 += SB) {
      constexpr int ROWS = 8 * (SB < BLOCKS ? SB : BLOCKS);
      if (a.bulk) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the last lines are read
      __syncwarp();
#pragma unroll
      for (int b = b0; b < b0 + SB && b < BLOCKS; b++) {
        const uint32_t sg = neg[8 * b + r];
        const auto val = [&](double x) { return (T)__hiloint2double(__double2hiint(x) ^ (int)sg, __double2loint(x)); };
        using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
        T* row = stage + (8 * (b - b0) + r) * 16 + 2 * q;
        *reinterpret_cast<V*>(row) = V{val(acc0[2 * b]), val(acc0[2 * b + 1])};
        *reinterpret_cast<V*>(row + 8) = V{val(acc1[2 * b]), val(acc1[2 * b + 1])};
      }
      const int* to = tgt + 8 * b0;
      if (a.bulk) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane < ROWS && to[lane] >= 0)
          bulk_add(a.S + (size_t)to[lane] * a.nb + ib0, smem_addr(stage + lane * 16),
                   (uint32_t)min((size_t)16, a.nb - ib0) * (uint32_t)sizeof(T));
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      } else {
        __syncwarp();
        const size_t ib = ib0 + (lane & 15);
#pragma unroll 4
        for (int row = lane >> 4; row < ROWS; row += 2)
          if (to[row] >= 0 && ib < a.nb) atomicAdd(a.S + (size_t)to[row] * a.nb + ib, stage[row * 16 + (lane & 15)]);
      }
    }
  }
  if (a.bulk) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// One CTA per (source alpha string ja, M of its singles): alpha single 8 b + r
// is row r of block b.
//
// With Ja, one more row per ja, with ja itself as its target, takes the beta
// singles' Coulomb parts sum_jb s_b J_rs[ja] C[ja,jb]: its integrals are J_rs[ja].
// As a pass of its own over the beta singles, between two transposes, that
// took 7.3 ms at 144M determinants; the row adds 1.6 % to the products.  (The
// alpha singles' Coulomb part J_pq[ib] C[ja,ib] as the value a row's sums start
// from cost 20 ms more, 5.4 against 4.0 ms at 16M: its loads stall the warps and
// take shared-memory wavefronts.  It stays a pass of its own.)
template <typename T, int M, int SB>
__global__ void __launch_bounds__(kMmaThreads) ab_mma_kernel(const MmaArgs<T> a) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int tgt[M];
  __shared__ uint32_t neg[M];
  unsigned char* vsub = smem;                                                          // [npair][M] integrals
  T* stage = reinterpret_cast<T*>(smem + (size_t)a.npair * M * 8);                     // [warps][8 SB][16] results
  double* crow = reinterpret_cast<double*>(stage + (size_t)(blockDim.x >> 5) * SB * 128);  // [nb + 1]
  const size_t ja = blockIdx.x;
  const int64_t k0 = a.a_off[ja] + (int64_t)blockIdx.y * M;
  const int singles = (int)min((int64_t)M, a.a_off[ja + 1] - k0);  // negative past the last ones
  if (singles < 0) return;
  const int count = singles + (a.Ja && singles < M ? 1 : 0);  // the row of ja itself comes after its last single
  if (count == 0) return;
  if (threadIdx.x < M) {
    const int g = threadIdx.x;
    tgt[g] = g < singles ? (int)((int64_t)a.a_idx[k0 + g] - (int64_t)a.ia0) : g < count ? (int)ja : -1;
    const uint32_t info = g < singles ? a.a_info[k0 + g] : 0u;
    neg[g] = info & 0x80000000u;
  }
  for (size_t i = threadIdx.x; i <= a.nb; i += blockDim.x) crow[i] = i < a.nb ? (double)a.C[ja * a.nb + i] : 0.0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  // one 32-byte chunk of eight pairs' rows per warp and step
  for (int c = 0; c < M / 4; c++) {
    const int place = 4 * c + (lane & 3);
    const int g = M == 16 ? 8 * (place & 1) + (place >> 1) : place;
    const double* vrow = g < singles ? a.vf + (size_t)((a.a_info[k0 + g] >> 12) & 0xFFFu) * a.P
                         : g < count ? a.Ja + ja
                                     : nullptr;
    const size_t step = g < singles ? 1 : a.na;
    for (int o = warp * 8 + (lane >> 2); o < a.npair; o += nwarp * 8)
      *reinterpret_cast<double*>(vsub + store_offset<M>(o, place)) =
          vrow ? __ldg(&vrow[(size_t)folded_pair(o) * step]) : 0.0;
  }
  __syncthreads();
  T* mine = stage + (size_t)warp * SB * 128;
  const unsigned char* cr = reinterpret_cast<const unsigned char*>(crow);
  if (M == 16 && count > 8)
    tiles<T, M, M / 8, SB>(a, vsub, cr, mine, tgt, neg);
  else
    tiles<T, M, 1, SB>(a, vsub, cr, mine, tgt, neg);
}

}  // namespace

namespace {

// dynamic shared memory: integrals, per-warp stages, the row of C
size_t mma_smem(const sbdgpu_ctx* c, int m, int threads, size_t elem, int sb) {
  return sizeof(double) * ((size_t)(c->L * (c->L - 1) / 2) * m + (c->nb + 1)) + elem * (threads / 32) * sb * 128;
}

template <typename T, int M, int SB>
void launch_mma(sbdgpu_ctx* c, const T* C, T* S, const AlphaSingles& as, int nt, bool beta_j) {
  const SpinTables& tb = c->tab[1];
  const dim3 grid((unsigned)c->na, (unsigned)((as.max_s + (beta_j ? 1 : 0) + M - 1) / M));
  if (grid.y == 0) return;
  // whole lines of sigma for the copy engine: 16-byte starts
  const int bulk = c->nb * sizeof(T) % 16 == 0 && ((uintptr_t)S & 15) == 0;
  const MmaArgs<T> a{C,
                  S,
                  c->na,
                  c->nb,
                  as.ia0,
                  c->P,
                  c->L * (c->L - 1) / 2,
                  c->vf,
                  as.off,
                  as.idx,
                  as.info,
                  tb.tile_grp,
                  tb.tile_ent,
                  (int)tb.n_tile_grp,
                  bulk,
                  beta_j ? c->ja : nullptr};
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<T, M, SB>), c->device);
  ab_mma_kernel<T, M, SB><<<grid, nt, mma_smem(c, M, nt, sizeof(T), SB), c->stream>>>(a);
  SBD_CUDA(cudaGetLastError());
}

}  // namespace

// Tiles of the beta singles for ab_mma_kernel.  A string given twice would put
// two kets into one slot, and the slots hold 16-bit kets with one value free
// for the zero: such bases keep the gather kernel.
void build_ab_tiles(sbdgpu_ctx* c, SpinTables& t, const std::vector<uint64_t>& strs) {
  const size_t n = strs.size();
  if (n == 0 || n > 65535) return;
  std::vector<uint64_t> sorted(strs);
  std::sort(sorted.begin(), sorted.end());
  if (std::adjacent_find(sorted.begin(), sorted.end()) != sorted.end()) return;
  for (uint64_t s : strs)
    if (__builtin_popcountll(s) != __builtin_popcountll(strs[0])) return;
  cudaStream_t st = c->stream;
  const int npair = c->L * (c->L - 1) / 2, words = (npair + 31) / 32;
  t.n_tile_grp = (n + 15) / 16;
  t.tile_grp = (int4*)dev_alloc(sizeof(int4) * t.n_tile_grp);
  tile_count_kernel<<<(unsigned)t.n_tile_grp, 32, 0, st>>>((int)n, words, t.s_off, t.s_info, t.tile_grp);
  SBD_CUDA(cudaGetLastError());
  std::vector<int4> h(t.n_tile_grp);
  SBD_CUDA(cudaMemcpyAsync(h.data(), t.tile_grp, sizeof(int4) * h.size(), cudaMemcpyDeviceToHost, st));
  SBD_CUDA(cudaStreamSynchronize(st));
  int64_t at = 0;
  for (auto& d : h) {
    d.x = (int)at;
    at += 2 * d.y + d.z + d.w;
  }
  t.tile_ent = (uint32_t*)dev_alloc(sizeof(uint32_t) * 32 * std::max<int64_t>(at, 1));
  SBD_CUDA(cudaMemcpyAsync(t.tile_grp, h.data(), sizeof(int4) * h.size(), cudaMemcpyHostToDevice, st));
  tile_fill_kernel<<<(unsigned)t.n_tile_grp, 32, 0, st>>>((int)n, words, t.s_off, t.s_idx, t.s_info, t.tile_grp,
                                                         t.tile_ent);
  SBD_CUDA(cudaGetLastError());
  SBD_CUDA(cudaStreamSynchronize(st));
}

// Alpha singles per CTA of the tile kernel for a wanted number (0: the larger
// that fits); 0 when this basis has no tiles or they do not fit.
int ab_mma_group(const sbdgpu_ctx* c, int want, size_t budget) {
  if (!c->tab[1].tile_grp) return 0;
  for (int m : {16, 8})
    if ((want == 0 || want == m) && mma_smem(c, m, 128, sizeof(double), 1) <= budget) return m;
  return 0;
}

// The alpha-beta term by tiles, m alpha singles per CTA, nt threads (0: the
// default); beta_j: the beta singles' Coulomb part as well (whole vectors
// only).  Default threads: those that put most warps on an SM beside the shared
// memory they need (at equal warps the smaller CTA), fewer while the warps
// outnumber the groups; results are staged for one block of alpha singles at a
// time where that lets more warps in.  Alpha-beta ms: 16M determinants 6.0 at
// 256 threads, 4.6 at 512, 5.6 at 768; 1501 x 803 strings 0.40 at 128, 0.34 at
// 256, 0.37 at 512; 144M 93 at 768 with both blocks staged, 97 and 88.6 at 768
// and 1,024 with one (FP32 vectors: 82 at 768, 77 at 1,024).
template <typename T>
void ab_mma(sbdgpu_ctx* c, const T* C, T* S, const AlphaSingles& as, int m, int nt, size_t budget, bool beta_j) {
  int sb = m / 8;
  if (nt == 0) {
    int best = 0;
    for (int b = m / 8; b >= 1; b--)
      for (int t : {256, 512, 768, 1024}) {
        const size_t smem = mma_smem(c, m, t, sizeof(T), b);
        if (smem > budget) break;
        const int warps = (int)std::min<size_t>(228 * 1024 / (smem + 1024), 1024 / t) * (t / 32);
        if (warps > best) {
          best = warps;
          nt = t;
          sb = b;
        }
      }
    if (nt == 0) {
      nt = 128;
      sb = 1;
    }
    while (nt > 128 && (size_t)(nt / 2) >= c->tab[1].n_tile_grp * 32) nt /= 2;
  } else {  // a tuned number: as many stages as fit beside the row of C
    if (mma_smem(c, m, nt, sizeof(T), sb) > budget) sb = 1;
    while (nt > 128 && mma_smem(c, m, nt, sizeof(T), sb) > budget) nt -= 128;
  }
  if (m == 16 && sb == 2)
    launch_mma<T, 16, 2>(c, C, S, as, nt, beta_j);
  else if (m == 16)
    launch_mma<T, 16, 1>(c, C, S, as, nt, beta_j);
  else
    launch_mma<T, 8, 1>(c, C, S, as, nt, beta_j);
}

template void ab_mma<double>(sbdgpu_ctx*, const double*, double*, const AlphaSingles&, int, int, size_t, bool);
template void ab_mma<float>(sbdgpu_ctx*, const float*, float*, const AlphaSingles&, int, int, size_t, bool);

void preload_ab_mma(int device) {
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<double, 16, 2>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<double, 16, 1>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<double, 8, 1>), device);
}

}  // namespace sbdgpu
