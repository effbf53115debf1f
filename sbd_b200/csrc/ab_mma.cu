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
// Tiles (built once per context): runs of up to eight beta strings, two n8
// tiles to a group.  The pairs both tiles use come first (one load of the
// integrals feeds both), then those of the first tile alone, then those of the
// second, each section in whole k4 steps.  The integral rows are turned by
// their pair's class modulo 4, so that four pairs of different classes lie in
// different banks; the pairs of a section are dealt to its steps by class and
// by the banks of their kets.  One 32-bit entry per slot, in the order of the B
// fragment (lane = 4 n + k).  Behind the row of C stand 16 zeros, one per bank
// pair; the empty slots of a half-warp point at one that none of its kets
// collides with.
#include <algorithm>
#include <functional>
#include <type_traits>
#include <vector>

#include "device.cuh"
#include "internal.cuh"

namespace sbdgpu {

namespace {

constexpr int kMmaThreads = 1024;
constexpr int kZeros = 16;     // zeros behind the row of C, one in each pair of banks
constexpr int kMaxWords = 63;  // bitmap words of the off-diagonal pairs: 64 * 63 / 2 = 2016

__device__ __forceinline__ int od_pair(uint32_t info) {  // off-diagonal pair index of a single
  return sbdgpu::od_pair((int)(info & 63), (int)((info >> 6) & 63));
}

// The folded pair (diagonal ones included) of off-diagonal pair o: as many
// diagonal pairs as its larger orbital come before.
__device__ __forceinline__ int folded_pair(int o) { return o + od_larger(o); }

// unions[i][l] = pairs used by the strings i .. i + l (l < 8), one warp per i
__global__ void __launch_bounds__(32) union_kernel(int n, int words, const int64_t* __restrict__ s_off,
                                                  const uint32_t* __restrict__ s_info, uint16_t* __restrict__ unions) {
  __shared__ uint32_t bm[kMaxWords + 1];
  const int i = blockIdx.x, lane = threadIdx.x;
  for (int w = lane; w < words; w += 32) bm[w] = 0;
  __syncwarp();
  for (int l = 0; l < 8; l++) {
    if (i + l < n)
      for (int64_t k = s_off[i + l] + lane; k < s_off[i + l + 1]; k += 32) {
        const int o = od_pair(s_info[k]);
        atomicOr(&bm[o >> 5], 1u << (o & 31));
      }
    __syncwarp();
    int c = 0;
    for (int w = lane; w < words; w += 32) c += __popc(bm[w]);
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) unions[(size_t)i * 8 + l] = (uint16_t)c;
    __syncwarp();
  }
}

// Bitmaps of the pairs used by the two tiles of a group (pos: first string and
// the tiles' lengths, second << 8 | first).  Sections of the pairs: 0 both
// tiles, 1 the first alone, 2 the second alone.
__device__ __forceinline__ void tile_bitmaps(uint32_t (*bm)[kMaxWords + 1], int words, int2 pos,
                                             const int64_t* __restrict__ s_off, const uint32_t* __restrict__ s_info) {
  const int lane = threadIdx.x;
  for (int w = lane; w < words; w += 32) bm[0][w] = bm[1][w] = 0;
  __syncwarp();
  for (int t = 0; t < 2; t++) {
    const int i0 = pos.x + (t ? pos.y & 0xFF : 0), i1 = i0 + (t ? pos.y >> 8 : pos.y & 0xFF);
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
__global__ void __launch_bounds__(32) tile_count_kernel(int words, const int64_t* __restrict__ s_off,
                                                       const uint32_t* __restrict__ s_info,
                                                       const int2* __restrict__ pos, int4* __restrict__ grp) {
  __shared__ uint32_t bm[2][kMaxWords + 1];
  const int g = blockIdx.x, lane = threadIdx.x;
  tile_bitmaps(bm, words, pos[g], s_off, s_info);
  int c[3] = {0, 0, 0};
  for (int w = lane; w < words; w += 32)
    for (int s = 0; s < 3; s++) c[s] += __popc(section_word(bm, s, w));
  for (int o = 16; o; o >>= 1)
    for (int s = 0; s < 3; s++) c[s] += __shfl_xor_sync(0xffffffffu, c[s], o);
  if (lane == 0) grp[g] = make_int4(0, (c[0] + 3) / 4, (c[1] + 3) / 4, (c[2] + 3) / 4);
}

// Beta and alpha strings from which cuts and deals are planned.  Planning takes
// 0.5 to 0.8 ms of a first pass at 12,000 to 20,000 beta strings; with 100 alpha
// strings or fewer the alpha-beta term takes less than 0.9 ms, planned or not.
constexpr size_t kPlannedTiles = 2048, kPlannedSources = 128;

// Per pair of a group, while its steps are dealt out.
struct PairPlan {
  uint32_t bank[2];  // bank pair of each string's ket, 4 bits per string, per tile
  uint16_t set;      // strings that have the pair, 8 bits per tile
  uint16_t pair;
  int16_t place;     // in its section; -1: not yet
};

__global__ void __launch_bounds__(32) tile_fill_kernel(int n, int words, const int64_t* __restrict__ s_off,
                                                      const int32_t* __restrict__ s_idx,
                                                      const uint32_t* __restrict__ s_info,
                                                      const int2* __restrict__ gpos, const int4* __restrict__ grp,
                                                      uint32_t* __restrict__ ent, bool by_banks) {
  extern __shared__ PairPlan plan[];
  __shared__ uint32_t bm[2][kMaxWords + 1];
  __shared__ int pre[3][kMaxWords + 1];  // plan index of a section's first pair in a word
  __shared__ int base[4];
  const int g = blockIdx.x, lane = threadIdx.x;
  const int2 pos = gpos[g];
  tile_bitmaps(bm, words, pos, s_off, s_info);
  if (lane == 0) {
    int at = 0;
    for (int s = 0; s < 3; s++) {
      base[s] = at;
      for (int w = 0; w < words; w++) {
        pre[s][w] = at;
        at += __popc(section_word(bm, s, w));
      }
    }
    base[3] = at;
  }
  __syncwarp();
  const auto index = [&](int o, int s) {
    return pre[s][o >> 5] + __popc(section_word(bm, s, o >> 5) & ((1u << (o & 31)) - 1u));
  };
  const auto section_of = [&](int o, int t) { return (bm[1 - t][o >> 5] >> (o & 31)) & 1u ? 0 : 1 + t; };
  const auto for_entries = [&](auto&& f) {
    for (int t = 0; t < 2; t++)
      for (int nn = 0; nn < (t ? pos.y >> 8 : pos.y & 0xFF); nn++) {
        const int i = pos.x + (t ? pos.y & 0xFF : 0) + nn;
        for (int64_t k = s_off[i] + lane; k < s_off[i + 1]; k += 32) f(t, nn, s_idx[k], s_info[k]);
      }
  };
  for (int o = lane; o < words * 32; o += 32)
    for (int s = 0; s < 3; s++)
      if ((section_word(bm, s, o >> 5) >> (o & 31)) & 1u) plan[index(o, s)] = PairPlan{{0, 0}, 0, (uint16_t)o, -1};
  __syncwarp();
  if (!by_banks) {  // by class alone: one pair of each while the classes last
    for (int s = 0; s < 3; s++)
      for (int c = base[s] + lane; c < base[s + 1]; c += 32) {
        const int cl = plan[c].pair & 3;
        int rank = 0, of[4] = {0, 0, 0, 0};
        for (int x = base[s]; x < base[s + 1]; x++) {
          const int k = plan[x].pair & 3;
          rank += x < c && k == cl;
          of[k]++;
        }
        int at = 0;
        for (int k = 0; k < 4; k++) at += min(of[k], rank) + (k < cl && of[k] > rank);
        plan[c].place = (int16_t)at;
      }
    __syncwarp();
  } else {
    for_entries([&](int t, int nn, int32_t ket, uint32_t info) {
      const int o = od_pair(info);
      PairPlan& p = plan[index(o, section_of(o, t))];
      atomicOr(&p.bank[t], (uint32_t)(ket & 15) << (4 * nn));
    });
    __syncwarp();
    // the strings' bits: one lane per pair would race on the half-word, one string at a time does not
    for (int t = 0; t < 2; t++)
      for (int nn = 0; nn < (t ? pos.y >> 8 : pos.y & 0xFF); nn++) {
        const int i = pos.x + (t ? pos.y & 0xFF : 0) + nn;
        for (int64_t k = s_off[i] + lane; k < s_off[i + 1]; k += 32) {
          const int o = od_pair(s_info[k]);
          plan[index(o, section_of(o, t))].set |= (uint16_t)(1u << (8 * t + nn));
        }
        __syncwarp();
      }
    // Deal the pairs of a section to its steps: the first one left, then three
    // times the one whose integral row differs in class from the step's others
    // and whose kets share fewest banks with theirs (per tile and half-warp of
    // four strings).
    for (int s = 0; s < 3; s++) {
      const int b0 = base[s], cnt = base[s + 1] - b0;
      uint64_t load[4] = {0, 0, 0, 0};  // 4-bit counts of 16 bank pairs by (tile, half)
      unsigned classes = 0;
      for (int at = 0; at < cnt; at++) {
        if ((at & 3) == 0) {
          classes = 0;
          for (int h = 0; h < 4; h++) load[h] = 0;
        }
        uint32_t best = 0xFFFFFFFFu;
        for (int c = lane; c < cnt; c += 32) {
          const PairPlan& p = plan[b0 + c];
          if (p.place >= 0) continue;
          uint32_t cost = 0;
          if (at & 3) {
            cost = (classes >> (p.pair & 3)) & 1u ? 8 : 0;
            for (int h = 0; h < 4; h++)
              for (int x = 0; x < 4; x++)
                if ((p.set >> (4 * h + x)) & 1)
                  cost += (uint32_t)(load[h] >> (4 * ((p.bank[h >> 1] >> (4 * (4 * (h & 1) + x))) & 15))) & 15u;
          }
          best = min(best, cost << 16 | (uint32_t)c);
        }
        const int pick = (int)(__reduce_min_sync(0xffffffffu, best) & 0xFFFFu);
        const PairPlan p = plan[b0 + pick];
        classes |= 1u << (p.pair & 3);
        for (int h = 0; h < 4; h++) {
          for (int x = 0; x < 4; x++)
            if ((p.set >> (4 * h + x)) & 1)
              load[h] += 1ull << (4 * ((p.bank[h >> 1] >> (4 * (4 * (h & 1) + x))) & 15));
        }
        __syncwarp();
        if (lane == 0) plan[b0 + pick].place = (int16_t)at;
        __syncwarp();
      }
    }
  }
  const int4 d = grp[g];
  uint32_t* out = ent + (size_t)d.x * 32;
  const uint32_t zero = (uint32_t)n << 3;  // the zero behind the row of C
  const auto first_word = [](uint32_t ket, int o, bool neg) {
    return (neg ? 1u : 0u) | ket << 3 | (uint32_t)(o << 2 | (o & 3)) << 19;
  };
  const auto second_word = [](uint32_t ket, bool neg) { return ket << 3 | (neg ? 0x80000000u : 0u); };
  const int64_t total = 32ll * (2 * d.y + d.z + d.w);
  for (int64_t k = lane; k < total; k += 32) out[k] = zero;
  __syncwarp();
  // entry of beta string `nn` (0..7) of tile t at place `at` of section s
  const auto slot = [&](int s, int at, int nn, int t) {
    const int step = at >> 2, lane_of = nn * 4 + (at & 3);
    if (s == 0) return ((size_t)step * 32 + lane_of) * 2 + t;
    return (size_t)(2 * d.y + (s == 2 ? d.z : 0) + step) * 32 + lane_of;
  };
  // every slot of a pair names the pair (the A operand of the whole column)
  for (int s = 0; s < 3; s++)
    for (int c = base[s] + lane; c < base[s + 1]; c += 32)
      for (int nn = 0; nn < 8; nn++)
        out[slot(s, plan[c].place, nn, 0)] = first_word((uint32_t)n, plan[c].pair, false);
  __syncwarp();
  for_entries([&](int t, int nn, int32_t ket, uint32_t info) {
    const int o = od_pair(info), s = section_of(o, t), at = plan[index(o, s)].place;
    const bool neg = info >> 31;
    out[slot(s, at, nn, t)] =
        s == 0 && t == 1 ? second_word((uint32_t)ket, neg) : first_word((uint32_t)ket, o, neg);
  });
  __syncwarp();
  // The empty slots of a half-warp read the zero whose bank none of its kets has
  // (one zero for all: 16M determinants 4.38 -> 4.31 ms, 144M 87.1 -> 85.1, FP32
  // vectors 74.4 -> 72.6).
  for (int u = lane; u < 2 * (2 * d.y + d.z + d.w); u += 32) {
    const bool both = u < 4 * d.y;
    uint32_t* w = both ? out + (u >> 2) * 64 + (u & 1) * 32 + ((u >> 1) & 1) : out + (size_t)u * 16;
    const int stride = both ? 2 : 1;
    uint32_t used = 0, empty = 0;
    for (int i = 0; i < 16; i++) {
      const uint32_t ket = (w[i * stride] >> 3) & 0xFFFFu;
      if (ket == (uint32_t)n)
        empty |= 1u << i;
      else
        used |= 1u << (ket & 15);
    }
    if (!empty) continue;
    const uint32_t shift = (uint32_t)(__ffs(~used) - 1 - n) & 15u;
    for (int i = 0; i < 16; i++)
      if ((empty >> i) & 1) w[i * stride] += shift << 3;
  }
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
// What bounds it: the shared-memory pipe (16M determinants: 87 % of its
// wavefronts, the FP64 tensor pipe 62 % busy).  Alpha-beta term with the beta
// singles' Coulomb part, gather kernel (without it) -> tiles: 144M determinants
// 198 -> 84 ms, 16M 11.2 -> 4.3 ms, 1501 x 803 strings 0.85 -> 0.34 ms,
// 495 x 495 0.10 -> 0.07 ms.  24 and 32 alpha
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
  const int2* pos;
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

// two results of a staged row of len, at columns c, c + 1
template <typename T>
__device__ __forceinline__ void put2(T* row, int c, int len, T x, T y) {
  using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  T* to = row + c;
  if (c + 1 < len && ((uintptr_t)to & (sizeof(V) - 1)) == 0) {
    *reinterpret_cast<V*>(to) = V{x, y};
  } else {
    if (c < len) to[0] = x;
    if (c + 1 < len) to[1] = y;
  }
}

// The groups of two tiles of one warp.  stage: the warp's [8 SB][16] results of
// SB blocks of alpha singles, whose rows are added to sigma as whole lines: by
// the copy engine where they start on 16 bytes, else by coalesced atomics.  (Added
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
    const int2 at = __ldg(&a.pos[g]);
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
    // the tiles' strings side by side: at.x .. at.x + len0 + len1
    const int len0 = at.y & 0xFF, len1 = at.y >> 8, len = len0 + len1;
    const bool bulk = a.bulk && (at.x * sizeof(T)) % 16 == 0 && (len * sizeof(T)) % 16 == 0;
    if constexpr (SB == 0) {  // no room for stages: straight from the accumulators
#pragma unroll
      for (int b = 0; b < BLOCKS; b++) {
        const int to = tgt[8 * b + r];
        if (to < 0) continue;
        const uint32_t sg = neg[8 * b + r];
        const auto val = [&](double x) { return (T)__hiloint2double(__double2hiint(x) ^ (int)sg, __double2loint(x)); };
        T* row = a.S + (size_t)to * a.nb + at.x;
#pragma unroll
        for (int u = 0; u < 2; u++) {
          if (2 * q + u < len0) atomicAdd(row + 2 * q + u, val(acc0[2 * b + u]));
          if (2 * q + u < len1) atomicAdd(row + len0 + 2 * q + u, val(acc1[2 * b + u]));
        }
      }
    } else {
#pragma unroll
      for (int b0 = 0; b0 < BLOCKS; b0 += SB) {
        constexpr int ROWS = 8 * (SB < BLOCKS ? SB : BLOCKS);
        if (a.bulk) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the last lines are read
        __syncwarp();
#pragma unroll
        for (int b = b0; b < b0 + SB && b < BLOCKS; b++) {
          const uint32_t sg = neg[8 * b + r];
          const auto val = [&](double x) { return (T)__hiloint2double(__double2hiint(x) ^ (int)sg, __double2loint(x)); };
          T* row = stage + (8 * (b - b0) + r) * 16;
          put2(row, 2 * q, len0, val(acc0[2 * b]), val(acc0[2 * b + 1]));
          put2(row + len0, 2 * q, len1, val(acc1[2 * b]), val(acc1[2 * b + 1]));
        }
        const int* to = tgt + 8 * b0;
        if (bulk) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane < ROWS && to[lane] >= 0)
            bulk_add(a.S + (size_t)to[lane] * a.nb + at.x, smem_addr(stage + lane * 16),
                     (uint32_t)len * (uint32_t)sizeof(T));
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        } else {
          __syncwarp();
          const int col = lane & 15;
#pragma unroll 4
          for (int row = lane >> 4; row < ROWS; row += 2)
            if (to[row] >= 0 && col < len) atomicAdd(a.S + (size_t)to[row] * a.nb + at.x + col, stage[row * 16 + col]);
        }
      }
    }
  }
  if (SB > 0 && a.bulk) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
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
  double* crow = reinterpret_cast<double*>(stage + (size_t)(blockDim.x >> 5) * SB * 128);  // [nb + kZeros]
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
  for (size_t i = threadIdx.x; i < a.nb + kZeros; i += blockDim.x) crow[i] = i < a.nb ? (double)a.C[ja * a.nb + i] : 0.0;
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
  return sizeof(double) * ((size_t)(c->L * (c->L - 1) / 2) * m + (c->nb + kZeros)) + elem * (threads / 32) * sb * 128;
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
                  tb.tile_pos,
                  tb.tile_ent,
                  (int)tb.n_tile_grp,
                  bulk,
                  beta_j ? c->ja : nullptr};
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<T, M, SB>), c->device);
  ab_mma_kernel<T, M, SB><<<grid, nt, mma_smem(c, M, nt, sizeof(T), SB), c->stream>>>(a);
  SBD_CUDA(cudaGetLastError());
}

}  // namespace

namespace {

void build_tiles(sbdgpu_ctx* c, SpinTables& t, const std::vector<uint64_t>& strs) {
  const size_t n = strs.size();
  if (n == 0 || n + kZeros > 65536) return;
  if (std::adjacent_find(strs.begin(), strs.end(), std::greater_equal<uint64_t>()) != strs.end()) {  // not ascending
    std::vector<uint64_t> sorted(strs);
    std::sort(sorted.begin(), sorted.end());
    if (std::adjacent_find(sorted.begin(), sorted.end()) != sorted.end()) return;
  }
  for (uint64_t s : strs)
    if (__builtin_popcountll(s) != __builtin_popcountll(strs[0])) return;
  // an infinite integral times the zero of an empty slot would be a NaN
  if (!c->vf_finite) return;
  cudaStream_t st = c->stream;
  const int npair = c->L * (c->L - 1) / 2, words = (npair + 31) / 32;
  // Tiles: runs of up to eight strings, cut where the union of their pairs would
  // jump (the runs of ascending strings that share their high orbitals are
  // rarely multiples of eight).  The cut with the fewest k4 steps, one more per
  // tile for its results, over all cuts at even strings (any, where an odd row
  // of sigma has no 16-byte lines to keep): 53 -> 58 % of the slots are filled at
  // 4,000 strings of 26 orbitals.
  std::vector<int> cut;  // first strings, then n
  const bool large = n >= kPlannedTiles && c->na >= kPlannedSources;
  if (!large) {
    for (size_t i = 0; i < n; i += 8) cut.push_back((int)i);
    cut.push_back((int)n);
  } else {
    uint16_t* d_u = (uint16_t*)dev_alloc(sizeof(uint16_t) * 8 * n);
    std::vector<uint16_t> u(8 * n);
    union_kernel<<<(unsigned)n, 32, 0, st>>>((int)n, words, t.s_off, t.s_info, d_u);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(u.data(), d_u, sizeof(uint16_t) * u.size(), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_u);
    SBD_CUDA(e);
    const size_t step = n % 2 ? 1 : 2;
    std::vector<int> best(n + 1, INT32_MAX), from(n + 1, 0);
    best[0] = 0;
    for (size_t i = 0; i < n; i += step)
      for (size_t l = step; l <= 8 && i + l <= n; l += step) {
        const int cost = best[i] + (u[8 * i + l - 1] + 3) / 4 + 1;
        if (cost < best[i + l]) {
          best[i + l] = cost;
          from[i + l] = (int)i;
        }
      }
    for (int i = (int)n; i > 0; i = from[i]) cut.push_back(i);
    cut.push_back(0);
    std::reverse(cut.begin(), cut.end());
  }
  const size_t ntile = cut.size() - 1;
  t.n_tile_grp = (ntile + 1) / 2;
  std::vector<int2> pos(t.n_tile_grp);
  for (size_t g = 0; g < pos.size(); g++) {
    const int a = cut[2 * g], b = cut[2 * g + 1], e = 2 * g + 2 <= ntile ? cut[2 * g + 2] : b;
    pos[g] = make_int2(a, (b - a) | (e - b) << 8);
  }
  t.tile_grp = (int4*)dev_alloc((sizeof(int4) + sizeof(int2)) * t.n_tile_grp);
  t.tile_pos = reinterpret_cast<int2*>(t.tile_grp + t.n_tile_grp);
  SBD_CUDA(cudaMemcpyAsync(t.tile_pos, pos.data(), sizeof(int2) * pos.size(), cudaMemcpyHostToDevice, st));
  tile_count_kernel<<<(unsigned)t.n_tile_grp, 32, 0, st>>>(words, t.s_off, t.s_info, t.tile_pos, t.tile_grp);
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
  tile_fill_kernel<<<(unsigned)t.n_tile_grp, 32, sizeof(PairPlan) * std::max(npair, 1), st>>>(
      (int)n, words, t.s_off, t.s_idx, t.s_info, t.tile_pos, t.tile_grp, t.tile_ent, large);
  SBD_CUDA(cudaGetLastError());
  SBD_CUDA(cudaStreamSynchronize(st));
}

}  // namespace

// Tiles of the beta singles for ab_mma_kernel.  A string given twice would put
// two kets into one slot, the slots hold 16-bit kets with sixteen values free
// for the zeros, and the integrals of a step meet strings without its pairs:
// bases of repeated or too many strings and non-finite integrals keep the
// gather kernel, and so does one whose tiles device memory has no room for.
void build_ab_tiles(sbdgpu_ctx* c, SpinTables& t, const std::vector<uint64_t>& strs) {
  try {
    build_tiles(c, t, strs);
  } catch (const Error& e) {
    if (e.code != SBDGPU_ERR_ALLOC) throw;
    cudaFree(t.tile_grp);
    cudaFree(t.tile_ent);
    t.tile_grp = nullptr;
    t.tile_pos = nullptr;
    t.tile_ent = nullptr;
    t.n_tile_grp = 0;
  }
}

// Without stages the kernel may use all that the opt-in limit leaves beside its
// own 128 bytes (budget is the limit less 1 KiB): eight singles beside 20,000
// beta strings at norb 48, where 490 ms replace the 1,180 ms of the gather
// kernel at four singles (400M determinants; FP32: 446 ms).
constexpr size_t kUnstagedExtra = 1024 - 128;

// Launch shape of the tile kernel for vectors of elem bytes.  group, threads:
// what the context was tuned to (0, 0: the default).  m = 0 when this basis has
// no tiles or they do not fit.
//
// Default: what bounds the kernel below some 24 warps per SM is latency, so the
// shape with most warps beside the shared memory they need (at equal warps the
// smaller CTA, with more stages); sixteen singles per CTA while 24 warps fit with
// them, else eight, without stages where that lets more warps in.  Alpha-beta ms
// at 16 singles and 24, 16, 8, 4 warps against 8 singles and 32 warps: 300 x
// 15,000 strings at norb 36 0.98 against 1.12, 16,500 1.29 against 1.20, 17,200
// 2.24 against 1.20, 17,900 4.28 against 1.18 (gather kernel 3.3).  Eight singles,
// 24 and 4 warps with stages against 32 without: 200 x 16,500 strings at norb 48
// 1.09 against 1.01, 19,300 6.06 against 1.20 (gather kernel 2.9).  Fewer threads
// while the warps outnumber the groups of beta strings and the eights of
// integral rows that they load: 20,000 x 40 strings at norb 36 10.6 ms at 128
// threads, 4.2 at 512 (gather kernel 9.9, FP32 4.8).
// Whole bases: 16M determinants 6.0 at 256 threads, 4.2 at 512, 5.0 at 768; 1501 x
// 803 strings 0.40 at 128, 0.34 at 256, 0.37 at 512; 144M 93 at 768 with both
// blocks staged, 97 and 88.6 at 768 and 1,024 with one (FP32 vectors: 82 at 768,
// 77 at 1,024).
MmaShape ab_mma_shape(const sbdgpu_ctx* c, int group, int threads, size_t elem, size_t budget) {
  if (!c->tab[1].tile_grp) return {};
  if (group > 0) {  // as many stages as fit beside the row of C
    MmaShape s{group, threads, group / 8};
    if ((group != 16 && group != 8) || mma_smem(c, group, 128, sizeof(double), 1) > budget) return {};
    if (mma_smem(c, group, s.nt, elem, s.sb) > budget) s.sb = 1;
    while (s.nt > 128 && mma_smem(c, group, s.nt, elem, s.sb) > budget) s.nt -= 128;
    return s;
  }
  MmaShape s;
  int best = 0;
  for (int m : {16, 8}) {
    for (int sb = m / 8; sb >= (m == 8 ? 0 : 1); sb--)
      for (int t : {256, 512, 768, 1024}) {
        const size_t smem = mma_smem(c, m, t, elem, sb);
        if (smem > budget + (sb == 0 ? kUnstagedExtra : 0)) break;
        const int warps = (int)std::min<size_t>(kSmemPerSM / (smem + 1024), 1024 / t) * (t / 32);
        if (warps > best) {
          best = warps;
          s = {m, t, sb};
        }
      }
    if (best >= 24) break;
    if (m == 16) best = 0;  // eight singles fit wherever sixteen do, with no fewer warps
  }
  const size_t loads = (size_t)(c->L * (c->L - 1) / 2 + 7) / 8;
  while (s.nt > 128 && (size_t)(s.nt / 2) >= 32 * std::max(c->tab[1].n_tile_grp, loads)) s.nt /= 2;
  return s;
}

// The alpha-beta term by tiles; beta_j: the beta singles' Coulomb part as well
// (whole vectors only).
template <typename T>
void ab_mma(sbdgpu_ctx* c, const T* C, T* S, const AlphaSingles& as, const MmaShape& s, bool beta_j) {
  if (s.m == 16 && s.sb == 2)
    launch_mma<T, 16, 2>(c, C, S, as, s.nt, beta_j);
  else if (s.m == 16)
    launch_mma<T, 16, 1>(c, C, S, as, s.nt, beta_j);
  else if (s.sb == 1)
    launch_mma<T, 8, 1>(c, C, S, as, s.nt, beta_j);
  else
    launch_mma<T, 8, 0>(c, C, S, as, s.nt, beta_j);
}

template void ab_mma<double>(sbdgpu_ctx*, const double*, double*, const AlphaSingles&, const MmaShape&, bool);
template void ab_mma<float>(sbdgpu_ctx*, const float*, float*, const AlphaSingles&, const MmaShape&, bool);

void preload_ab_mma(int device) {
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<double, 16, 2>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<double, 16, 1>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<double, 8, 1>), device);
  allow_dynamic_smem(reinterpret_cast<const void*>(ab_mma_kernel<double, 8, 0>), device);
}

}  // namespace sbdgpu
