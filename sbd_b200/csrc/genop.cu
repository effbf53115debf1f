// The generic path: a second-quantised operator (basic/generalop.h GeneralOp)
// applied to a vector on a basis of bit strings (basic/basis.h Basis), and the
// Lanczos and Davidson solvers built on it (basic/out_of_place_func/mult.h,
// lanczos.h, davidson.h), at one rank on one GPU.
//
// Layout in HBM:
//   states      [n][nw] uint64 in the caller's order (site q at bit q%64 of
//               word q/64), nw = 1, 2 or 4
//   hash table  open addressing with linear probing over a power-of-two table
//               of at least four times the states (twice above 1 GiB): a slot
//               holds the key words and, during a mult, the state's vector
//               element, so that one probe returns the value itself (a slot of
//               one-word states is 16 bytes: one sector per term instead of
//               three for index, key and element).  An empty slot's key is a configuration outside the
//               basis and its element 0.
//   terms       the off-diagonal list as arrays (creation mask, sign mask,
//               coefficient) sorted by annihilation mask, with one bucket
//               record per distinct mask; the diagonal list is folded into one
//               number per state at set-up (hdiag)
//
// mult: one warp per bra state.  Its lanes test 32 buckets at a time for
// annihilated sites that are all occupied in the state and split the terms of
// each bucket that passes.  A term applies when its created sites are empty
// after the annihilation, which with the bucket's test is the reference's
// sequential test (mult.h:213-240) for terms whose annihilated sites are
// distinct and whose created sites are distinct (a term that repeats a site in
// either part never applies there and is dropped at set-up).  The sign is the
// parity of the occupied sites below each operator's site, in order: the
// operators before it have flipped sites of their own, so the total is the
// parity of the state under the exclusive-or of the "below" masks, times a
// constant that goes into the coefficient.  The lanes' sums are reduced in the
// warp, so no atomics.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <iostream>
#include <mutex>
#include <numeric>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "internal.cuh"

using sbdgpu::Error;

struct sbdgpu_genop {
  sbdgpu_ctx base;  // device, stream, reduction scratch and the error string
  int nw = 1;
  size_t n = 0;
  int sign = 1;
  uint64_t* states = nullptr;
  void* slots = nullptr;      // hash table, Slot<nw> each
  std::mutex mult_mu;         // the slots' elements belong to one mult at a time, from its scatter on
  int64_t* slot_of = nullptr; // [n] slot of every state
  uint64_t hmask = 0;         // slots - 1
  uint64_t absent[4] = {};    // key of an empty slot: a configuration outside the basis
  uint64_t site_or[4] = {};   // every site of a basis state
  uint64_t term_or[4] = {};   // every site an off-diagonal term creates
  // off-diagonal terms, sorted by annihilation mask
  uint64_t* t_cre = nullptr;   // [n_terms][nw] created sites
  uint64_t* t_sgn = nullptr;   // [n_terms][nw] sites whose occupations give the sign
  double* t_coef = nullptr;    // coefficient, the sign's constant part included
  void* buckets = nullptr;     // one record per distinct annihilation mask
  size_t n_buckets = 0;
  size_t n_terms = 0;
  void* self_terms = nullptr;  // off-diagonal records that map a state onto itself
  size_t n_self = 0;
  double* hdiag = nullptr;     // diagonal list, per state (caller order)
  bool ready = false;
};

namespace {

constexpr int kMaxOps = SBDGPU_GENOP_MAX_OPS;
constexpr int kThreads = 256;

template <int NW>
struct Term {
  uint64_t ann[NW];
  uint64_t cre[NW];
  double coef;
  int32_t nops, ndag;
  uint8_t site[kMaxOps];
};

template <int NW>
struct DiagTerm {
  uint64_t mask[NW];
  double coef;
};

template <int NW>
struct Bucket {
  uint64_t ann[NW];
  int64_t start, end;  // its terms in the sorted term array
};

// Hash of a state, in 32-bit steps: two odd multipliers per word, then one
// round of shifts and a multiply, enough to spread bit strings that differ in a
// few sites (at a quarter full: 1.15 probes per search, 97 % within two).  The
// upper half only serves tables of more than 2^32 slots.  Multipliers: xxHash's
// first three 32-bit primes, and one of C. Wellons's hash prospector.
template <int NW>
__host__ __device__ __forceinline__ uint64_t hash_state(const uint64_t* w, uint64_t hmask) {
  uint32_t h = 0;
  for (int x = 0; x < NW; x++) {
    h = (h ^ (h >> 16)) + (uint32_t)w[x] * 0x9E3779B1u + (uint32_t)(w[x] >> 32) * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
  }
  uint64_t r = h ^ (h >> 13);
  if (hmask >> 32) r |= (uint64_t)((uint32_t)(w[0] >> 16) * 0xC2B2AE3Du ^ h) << 32;
  return r & hmask;
}

template <int NW>
struct alignas(NW == 1 ? 16 : NW == 2 ? 32 : 64) Slot {
  uint64_t key[NW];
  double val;
};

template <int NW>
struct Words {
  uint64_t w[NW];
};

// The off-diagonal terms on the device.
template <int NW>
struct TermList {
  const Bucket<NW>* buckets;
  size_t n_buckets;
  const uint64_t* cre;
  const uint64_t* sgn;
  const double* coef;
};

// acc += c * (the vector element of state w), nothing when w is outside the
// basis (not c times zero: c may be infinite)
template <int NW>
__device__ __forceinline__ void add_element(const Slot<NW>* __restrict__ slots, uint64_t hmask, const uint64_t* absent,
                                            const uint64_t* w, double c, double& acc) {
  uint64_t h = hash_state<NW>(w, hmask);
  // the table is at most half full, so an empty slot ends every probe
  // sequence; the bound keeps the loop finite regardless
  for (uint64_t probe = 0; probe <= hmask; probe++) {
    uint64_t key[NW];
    double val;
    if constexpr (NW == 1) {
      const ulonglong2 x = __ldg(reinterpret_cast<const ulonglong2*>(&slots[h]));
      key[0] = x.x;
      val = __longlong_as_double((long long)x.y);
    } else {
#pragma unroll
      for (int x = 0; x < NW; x++) key[x] = __ldg(&slots[h].key[x]);
      val = __ldg(&slots[h].val);
    }
    bool eq = true, empty = true;
#pragma unroll
    for (int x = 0; x < NW; x++) {
      eq &= key[x] == w[x];
      empty &= key[x] == absent[x];
    }
    if (empty) return;
    if (eq) {
      acc += c * val;
      return;
    }
    h = (h + 1) & hmask;
  }
}

// slots' elements <- C
template <int NW>
__global__ void scatter_kernel(Slot<NW>* __restrict__ slots, const int64_t* __restrict__ slot_of,
                               const double* __restrict__ C, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    slots[slot_of[i]].val = C[i];
}

// Calls f(lane applies, target, coefficient with sign) for every term of every
// bucket that applies to state v, by the whole warp (lanes past a bucket's end
// or whose term does not apply are called with false).
template <int NW, class F>
__device__ __forceinline__ void for_terms(const TermList<NW>& tl, const uint64_t (&v)[NW], F&& f) {
  const int lane = threadIdx.x & 31;
  for (size_t b0 = 0; b0 < tl.n_buckets; b0 += 32) {
    bool ok = b0 + lane < tl.n_buckets;
    if (ok) {
#pragma unroll
      for (int x = 0; x < NW; x++) {
        const uint64_t m = __ldg(&tl.buckets[b0 + lane].ann[x]);
        ok &= (v[x] & m) == m;
      }
    }
    for (unsigned hits = __ballot_sync(0xffffffffu, ok); hits; hits &= hits - 1) {
      const Bucket<NW>* bk = &tl.buckets[b0 + __ffs((int)hits) - 1];
      uint64_t left[NW];
#pragma unroll
      for (int x = 0; x < NW; x++) left[x] = v[x] & ~__ldg(&bk->ann[x]);
      const int64_t t1 = __ldg(&bk->end);
      for (int64_t t0 = __ldg(&bk->start); t0 < t1; t0 += 32) {
        const int64_t t = t0 + lane;
        bool on = t < t1;
        uint64_t w[NW];
        double c = 0.0;
        if (on) {
          int par = 0;
#pragma unroll
          for (int x = 0; x < NW; x++) {
            const uint64_t cre = __ldg(&tl.cre[t * NW + x]);
            on &= (left[x] & cre) == 0ull;
            w[x] = left[x] | cre;
            par += __popcll(v[x] & __ldg(&tl.sgn[t * NW + x]));
          }
          c = __ldg(&tl.coef[t]);
          c = par & 1 ? -c : c;
        }
        f(on, w, c);
      }
    }
  }
}

// parity of the occupied sites below q
template <int NW>
__device__ __forceinline__ int parity_below(const uint64_t* w, int q) {
  int c = 0;
  const int r = q >> 6;
#pragma unroll
  for (int x = 0; x < NW; x++) {
    if (x < r) c += __popcll(w[x]);
    else if (x == r) c += __popcll(w[x] & ((1ull << (q & 63)) - 1ull));
  }
  return c & 1;
}

// Apply term t to state v: false when it does not apply; else the target in
// w and the sign (+1 or -1; +1 when sign is off).
template <int NW>
__device__ __forceinline__ bool apply_term(const Term<NW>& t, const uint64_t* v, int sign, uint64_t* w, double* s) {
  bool ok = true;
#pragma unroll
  for (int x = 0; x < NW; x++) {
    ok &= (v[x] & t.ann[x]) == t.ann[x];
    ok &= ((v[x] & ~t.ann[x]) & t.cre[x]) == 0ull;
  }
  if (!ok) return false;
  int par = 0;
  if (sign) {
#pragma unroll
    for (int x = 0; x < NW; x++) w[x] = v[x];
    for (int k = 0; k < t.nops; k++) {
      const int q = t.site[k];
      const uint64_t b = 1ull << (q & 63);
      if (k < t.ndag) w[q >> 6] &= ~b;
      else w[q >> 6] |= b;
      par ^= parity_below<NW>(w, q);
    }
  } else {
#pragma unroll
    for (int x = 0; x < NW; x++) w[x] = (v[x] & ~t.ann[x]) | t.cre[x];
  }
  *s = par ? -1.0 : 1.0;
  return true;
}

// W[i] += hdiag[i] C[i] + sum over off-diagonal terms of coef * sign * C[j]:
// one warp per state.  Bound by the integer pipe (81 % busy).  The 349M elements
// of the 245,025-state FCIDUMP operator: 16.1 ms with index, key and element in
// three sectors, the sign from the operators one by one and the buckets tested
// one after another; 6.6 ms with one sector, the sign by mask and 32 buckets at
// a time; 4.8 ms with a 32-bit hash and a quarter-full table; 4.6 ms with nothing
// added for targets outside the basis.  (Queueing the targets that apply and
// probing for 32 at a time: 4.9 against 4.8 ms.)
constexpr int kMultWarps = kThreads / 32;
template <int NW>
__global__ void __launch_bounds__(kThreads) mult_kernel(const uint64_t* __restrict__ states, size_t n,
                                                       const Slot<NW>* __restrict__ slots, uint64_t hmask,
                                                       Words<NW> absent, TermList<NW> tl,
                                                       const double* __restrict__ hdiag,
                                                       const double* __restrict__ C, double* __restrict__ W) {
  const int lane = threadIdx.x & 31;
  const size_t warps = (size_t)gridDim.x * kMultWarps;
  for (size_t i = (size_t)blockIdx.x * kMultWarps + (threadIdx.x >> 5); i < n; i += warps) {
    uint64_t v[NW];
#pragma unroll
    for (int x = 0; x < NW; x++) v[x] = __ldg(&states[i * NW + x]);
    double acc = 0.0;
    for_terms<NW>(tl, v, [&](bool on, const uint64_t (&w)[NW], double c) {
      if (on) add_element<NW>(slots, hmask, absent.w, w, c, acc);
    });
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) W[i] = W[i] + hdiag[i] * C[i] + acc;
  }
}

// hdiag[i] = sum of the diagonal terms whose sites are all occupied in state i
template <int NW>
__global__ void __launch_bounds__(kThreads) diag_kernel(const uint64_t* __restrict__ states, size_t n,
                                                       const DiagTerm<NW>* __restrict__ terms, size_t n_terms,
                                                       double* __restrict__ hdiag) {
  const size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  uint64_t v[NW];
#pragma unroll
  for (int x = 0; x < NW; x++) v[x] = states[i * NW + x];
  double acc = 0.0;
  for (size_t k = 0; k < n_terms; k++) {
    bool ok = true;
#pragma unroll
    for (int x = 0; x < NW; x++) ok &= (v[x] & terms[k].mask[x]) == terms[k].mask[x];
    if (ok) acc += terms[k].coef;
  }
  hdiag[i] = acc;
}

// out[i] = hdiag[i] + sum of the self-mapping off-diagonal terms that apply
template <int NW>
__global__ void __launch_bounds__(kThreads) self_kernel(const uint64_t* __restrict__ states, size_t n,
                                                       const Term<NW>* __restrict__ terms, size_t n_terms, int sign,
                                                       const double* __restrict__ hdiag, double* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  uint64_t v[NW];
#pragma unroll
  for (int x = 0; x < NW; x++) v[x] = states[i * NW + x];
  double acc = hdiag[i];
  for (size_t k = 0; k < n_terms; k++) {
    uint64_t w[NW];
    double s;
    if (apply_term<NW>(terms[k], v, sign, w, &s)) acc += terms[k].coef * s;
  }
  out[i] = acc;
}

unsigned blocks_for(size_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

template <class F>
int guarded(sbdgpu_genop* g, F&& f) {
  if (!g) return SBDGPU_ERR_ARG;
  try {
    cudaError_t e = cudaSetDevice(g->base.device);
    if (e != cudaSuccess) throw Error{SBDGPU_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e)};
    f();
    g->base.err.clear();
    return SBDGPU_OK;
  } catch (const Error& e) {
    g->base.err = e.msg;
    return e.code;
  } catch (const std::bad_alloc&) {
    g->base.err = "host allocation failed";
    return SBDGPU_ERR_ALLOC;
  } catch (const std::exception& e) {
    g->base.err = e.what();
    return SBDGPU_ERR_STATE;
  }
}

constexpr uint32_t kFree = 0xFFFFFFFFu;

// Every state claims the first free slot of its search: owner of a slot, slot
// of a state; *repeated is set where a search meets the state's own key.
template <int NW>
__global__ void insert_kernel(const uint64_t* __restrict__ states, size_t n, uint64_t hmask,
                              uint32_t* __restrict__ owner, int64_t* __restrict__ slot_of, int* __restrict__ repeated) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    uint64_t w[NW];
#pragma unroll
    for (int x = 0; x < NW; x++) w[x] = states[i * NW + x];
    uint64_t h = hash_state<NW>(w, hmask);
    for (uint64_t probe = 0; probe <= hmask; probe++, h = (h + 1) & hmask) {
      const uint32_t other = atomicCAS(&owner[h], kFree, (uint32_t)i);
      if (other == kFree) {
        slot_of[i] = (int64_t)h;
        break;
      }
      bool eq = true;
#pragma unroll
      for (int x = 0; x < NW; x++) eq &= states[(size_t)other * NW + x] == w[x];
      if (eq) {
        *repeated = 1;
        break;
      }
    }
  }
}

template <int NW>
__global__ void keys_kernel(const uint64_t* __restrict__ states, const uint32_t* __restrict__ owner, size_t count,
                            Words<NW> absent, Slot<NW>* __restrict__ slots) {
  for (size_t h = (size_t)blockIdx.x * blockDim.x + threadIdx.x; h < count; h += (size_t)gridDim.x * blockDim.x) {
    const uint32_t i = owner[h];
    Slot<NW> s;
#pragma unroll
    for (int x = 0; x < NW; x++) s.key[x] = i == kFree ? absent.w[x] : states[(size_t)i * NW + x];
    s.val = 0.0;
    slots[h] = s;
  }
}

// The basis on the device: states, hash table and every state's slot.  The
// table is filled there: 1,002,001 states take 4 ms, on the host they took 73-90
// ms (24-30 ms as a half-full table of keys and indices), most of it the
// table's cache misses and its copy.
template <int NW>
void build_basis(sbdgpu_genop* g, const uint64_t* states) {
  const size_t n = g->n;
  if (n >= kFree) throw Error{SBDGPU_ERR_ALLOC, "basis larger than device memory"};
  cudaStream_t st = g->base.stream;
  // a power of two of at least four times the states (twice above 1 GiB: the
  // lanes of a warp wait for their longest search)
  size_t count = 1024;
  while (count < 4 * n && (count < 2 * n || count * sizeof(Slot<NW>) < (size_t(1) << 30))) count <<= 1;
  g->hmask = count - 1;
  // the first configuration from the top that no state has
  std::vector<uint64_t> top;  // distances of the states near it
  for (size_t i = 0; i < n; i++) {
    bool high = true;
    for (int x = 0; x < NW; x++) {
      g->site_or[x] |= states[i * NW + x];
      high &= x == 0 || states[i * NW + x] == ~0ull;
    }
    if (high && ~states[i * NW] < n) top.push_back(~states[i * NW]);
  }
  std::sort(top.begin(), top.end());
  Words<NW> absent;
  std::fill(absent.w, absent.w + NW, ~0ull);
  for (uint64_t d : top)
    if (d == ~absent.w[0]) absent.w[0]--;
  std::memcpy(g->absent, absent.w, sizeof(absent.w));
  g->states = (uint64_t*)sbdgpu::dev_alloc(sizeof(uint64_t) * n * NW);
  g->slots = sbdgpu::dev_alloc(sizeof(Slot<NW>) * count);
  g->slot_of = (int64_t*)sbdgpu::dev_alloc(sizeof(int64_t) * n);
  sbdgpu::Arena arena(st);
  uint32_t* owner = nullptr;
  int* repeated = nullptr;
  arena.add(&owner, count);
  arena.add(&repeated, 1);
  arena.commit();
  SBD_CUDA(cudaMemcpyAsync(g->states, states, sizeof(uint64_t) * n * NW, cudaMemcpyHostToDevice, st));
  SBD_CUDA(cudaMemsetAsync(owner, 0xFF, sizeof(uint32_t) * count, st));
  SBD_CUDA(cudaMemsetAsync(repeated, 0, sizeof(int), st));
  const auto grid = [](size_t m) { return (unsigned)std::min<size_t>((m + kThreads - 1) / kThreads, 148 * 8); };
  insert_kernel<NW><<<grid(n), kThreads, 0, st>>>(g->states, n, g->hmask, owner, g->slot_of, repeated);
  SBD_CUDA(cudaGetLastError());
  keys_kernel<NW><<<grid(count), kThreads, 0, st>>>(g->states, owner, count, absent, static_cast<Slot<NW>*>(g->slots));
  SBD_CUDA(cudaGetLastError());
  int r = 0;
  SBD_CUDA(cudaMemcpyAsync(&r, repeated, sizeof(int), cudaMemcpyDeviceToHost, st));
  SBD_CUDA(cudaStreamSynchronize(st));
  if (r) throw Error{SBDGPU_ERR_ARG, "repeated basis state"};
}

// One list's terms as host records.  Off-diagonal terms that repeat a site
// among their annihilated or among their created operators never apply
// (the reference's sequential test fails at the repeat) and are left out.
template <int NW>
void build_terms(int nw, size_t n_terms, const int64_t* off, const int32_t* ops, const int32_t* ndag,
                 const double* coef, std::vector<Term<NW>>& all, std::vector<Term<NW>>& self) {
  const int max_site = 64 * nw;
  for (size_t k = 0; k < n_terms; k++) {
    const int64_t a = off[k], b = off[k + 1];
    if (b < a) throw Error{SBDGPU_ERR_ARG, "term offsets must not decrease"};
    const int nops = (int)(b - a);
    if (nops > kMaxOps) throw Error{SBDGPU_ERR_ARG, "more than " + std::to_string(kMaxOps) + " operators in a term"};
    if (ndag[k] < 0 || ndag[k] > nops) throw Error{SBDGPU_ERR_ARG, "n_dag out of range"};
    Term<NW> t;
    std::memset(&t, 0, sizeof(t));
    t.coef = coef[k];
    t.nops = nops;
    t.ndag = ndag[k];
    bool repeat = false;
    for (int j = 0; j < nops; j++) {
      const int q = ops[a + j] & 0xFFFF;
      if (q >= max_site) throw Error{SBDGPU_ERR_ARG, "site " + std::to_string(q) + " beyond the state width"};
      t.site[j] = (uint8_t)q;
      uint64_t* m = j < t.ndag ? t.ann : t.cre;
      const uint64_t bit = 1ull << (q & 63);
      if (m[q >> 6] & bit) repeat = true;
      m[q >> 6] |= bit;
    }
    if (repeat) continue;
    all.push_back(t);
    if (std::equal(t.ann, t.ann + NW, t.cre)) self.push_back(t);
  }
}

template <int NW>
void set_terms_nw(sbdgpu_genop* g, size_t n_diag, const int64_t* diag_off, const int32_t* diag_ops,
                  const int32_t* diag_ndag, const double* diag_coef, size_t n_off, const int64_t* off_off,
                  const int32_t* off_ops, const int32_t* off_ndag, const double* off_coef) {
  cudaStream_t st = g->base.stream;
  std::vector<DiagTerm<NW>> dt;
  dt.reserve(n_diag);
  for (size_t k = 0; k < n_diag; k++) {
    const int64_t a = diag_off[k], b = diag_off[k + 1];
    if (b < a) throw Error{SBDGPU_ERR_ARG, "term offsets must not decrease"};
    if (diag_ndag[k] < 0 || diag_ndag[k] > b - a) throw Error{SBDGPU_ERR_ARG, "n_dag out of range"};
    DiagTerm<NW> d;
    std::memset(&d, 0, sizeof(d));
    d.coef = diag_coef[k];
    for (int j = 0; j < diag_ndag[k]; j++) {  // the sites of the first n_dag operators (mult.h:130-139)
      const int q = diag_ops[a + j] & 0xFFFF;
      if (q >= 64 * NW) throw Error{SBDGPU_ERR_ARG, "site " + std::to_string(q) + " beyond the state width"};
      d.mask[q >> 6] |= 1ull << (q & 63);
    }
    dt.push_back(d);
  }
  std::vector<Term<NW>> all, self;
  build_terms<NW>(NW, n_off, off_off, off_ops, off_ndag, off_coef, all, self);
  // terms grouped by annihilation mask (stable), one bucket per mask
  std::stable_sort(all.begin(), all.end(), [](const Term<NW>& a, const Term<NW>& b) {
    return std::lexicographical_compare(a.ann, a.ann + NW, b.ann, b.ann + NW);
  });
  std::vector<Bucket<NW>> bk;
  for (size_t t = 0; t < all.size(); t++) {
    if (t == 0 || !std::equal(all[t].ann, all[t].ann + NW, all[t - 1].ann)) {
      Bucket<NW> b;
      std::memcpy(b.ann, all[t].ann, sizeof(b.ann));
      b.start = (int64_t)t;
      bk.push_back(b);
    }
    bk.back().end = (int64_t)t + 1;
  }
  // creation masks, sign masks (below-masks of the operators' sites) and
  // coefficients with the constant part of the sign: the operators before one
  // have flipped their own sites, those below it count
  std::vector<uint64_t> cre(all.size() * NW), sgn(all.size() * NW, 0);
  std::vector<double> cf(all.size());
  uint64_t term_or[4] = {};
  for (size_t t = 0; t < all.size(); t++) {
    int flips = 0;
    for (int k = 0; g->sign && k < all[t].nops; k++) {
      const int q = all[t].site[k];
      for (int x = 0; x < (q >> 6); x++) sgn[t * NW + x] ^= ~0ull;
      sgn[t * NW + (q >> 6)] ^= (1ull << (q & 63)) - 1ull;
      for (int j = 0; j < k; j++) flips += all[t].site[j] < q;
    }
    cf[t] = flips & 1 ? -all[t].coef : all[t].coef;
    for (int x = 0; x < NW; x++) {
      cre[t * NW + x] = all[t].cre[x];
      term_or[x] |= all[t].cre[x];
    }
  }
  std::memcpy(g->term_or, term_or, sizeof(term_or));
  cudaFree(g->t_cre);
  cudaFree(g->t_sgn);
  cudaFree(g->t_coef);
  cudaFree(g->self_terms);
  cudaFree(g->buckets);
  g->self_terms = g->buckets = nullptr;
  g->t_cre = g->t_sgn = nullptr;
  g->t_coef = nullptr;
  g->n_buckets = 0;
  g->ready = false;
  DiagTerm<NW>* d_dt = nullptr;
  try {
    if (!dt.empty()) {
      d_dt = (DiagTerm<NW>*)sbdgpu::dev_alloc(sizeof(DiagTerm<NW>) * dt.size());
      SBD_CUDA(cudaMemcpyAsync(d_dt, dt.data(), sizeof(DiagTerm<NW>) * dt.size(), cudaMemcpyHostToDevice, st));
    }
    if (!g->hdiag) g->hdiag = (double*)sbdgpu::dev_alloc(sizeof(double) * g->n);
    diag_kernel<NW><<<blocks_for(g->n), kThreads, 0, st>>>(g->states, g->n, d_dt, dt.size(), g->hdiag);
    SBD_CUDA(cudaGetLastError());
    if (!all.empty()) {
      const size_t mask_bytes = sizeof(uint64_t) * NW * all.size();
      g->t_cre = (uint64_t*)sbdgpu::dev_alloc(mask_bytes);
      SBD_CUDA(cudaMemcpyAsync(g->t_cre, cre.data(), mask_bytes, cudaMemcpyHostToDevice, st));
      g->t_sgn = (uint64_t*)sbdgpu::dev_alloc(mask_bytes);
      SBD_CUDA(cudaMemcpyAsync(g->t_sgn, sgn.data(), mask_bytes, cudaMemcpyHostToDevice, st));
      g->t_coef = (double*)sbdgpu::dev_alloc(sizeof(double) * all.size());
      SBD_CUDA(cudaMemcpyAsync(g->t_coef, cf.data(), sizeof(double) * all.size(), cudaMemcpyHostToDevice, st));
      g->buckets = sbdgpu::dev_alloc(sizeof(Bucket<NW>) * bk.size());
      SBD_CUDA(cudaMemcpyAsync(g->buckets, bk.data(), sizeof(Bucket<NW>) * bk.size(), cudaMemcpyHostToDevice, st));
    }
    if (!self.empty()) {
      g->self_terms = sbdgpu::dev_alloc(sizeof(Term<NW>) * self.size());
      SBD_CUDA(cudaMemcpyAsync(g->self_terms, self.data(), sizeof(Term<NW>) * self.size(), cudaMemcpyHostToDevice,
                               st));
    }
    SBD_CUDA(cudaStreamSynchronize(st));
  } catch (...) {
    cudaFree(d_dt);
    throw;
  }
  cudaFree(d_dt);
  g->n_terms = all.size();
  g->n_buckets = bk.size();
  g->n_self = self.size();
  g->ready = true;
}

template <int NW>
TermList<NW> term_list(const sbdgpu_genop* g) {
  return TermList<NW>{static_cast<const Bucket<NW>*>(g->buckets), g->n_buckets, g->t_cre, g->t_sgn, g->t_coef};
}

template <int NW>
void mult_nw(sbdgpu_genop* g, const double* C, double* W) {
  Slot<NW>* slots = static_cast<Slot<NW>*>(g->slots);
  // both launches in a row on the object's stream, whichever host threads call
  std::lock_guard<std::mutex> lock(g->mult_mu);
  scatter_kernel<NW><<<(unsigned)std::min<size_t>(blocks_for(g->n), 148 * 8), kThreads, 0, g->base.stream>>>(
      slots, g->slot_of, C, g->n);
  SBD_CUDA(cudaGetLastError());
  Words<NW> absent;
  std::memcpy(absent.w, g->absent, sizeof(absent.w));
  const unsigned grid = (unsigned)std::min<size_t>((g->n + kMultWarps - 1) / kMultWarps, 148 * 64);
  mult_kernel<NW><<<grid, kThreads, 0, g->base.stream>>>(g->states, g->n, slots, g->hmask, absent, term_list<NW>(g),
                                                        g->hdiag, C, W);
  SBD_CUDA(cudaGetLastError());
}

void mult(sbdgpu_genop* g, const double* C, double* W) {
  if (!g->ready) throw Error{SBDGPU_ERR_STATE, "no operator: call sbdgpu_genop_set_terms first"};
  switch (g->nw) {
    case 1: mult_nw<1>(g, C, W); break;
    case 2: mult_nw<2>(g, C, W); break;
    default: mult_nw<4>(g, C, W); break;
  }
}

void diagonal(sbdgpu_genop* g, double* out) {
  if (!g->ready) throw Error{SBDGPU_ERR_STATE, "no operator: call sbdgpu_genop_set_terms first"};
  cudaStream_t st = g->base.stream;
  switch (g->nw) {
    case 1:
      self_kernel<1><<<blocks_for(g->n), kThreads, 0, st>>>(g->states, g->n, static_cast<const Term<1>*>(g->self_terms),
                                                            g->n_self, g->sign, g->hdiag, out);
      break;
    case 2:
      self_kernel<2><<<blocks_for(g->n), kThreads, 0, st>>>(g->states, g->n, static_cast<const Term<2>*>(g->self_terms),
                                                            g->n_self, g->sign, g->hdiag, out);
      break;
    default:
      self_kernel<4><<<blocks_for(g->n), kThreads, 0, st>>>(g->states, g->n, static_cast<const Term<4>*>(g->self_terms),
                                                            g->n_self, g->sign, g->hdiag, out);
      break;
  }
  SBD_CUDA(cudaGetLastError());
}

struct DevVecs {
  std::vector<double*> p;
  cudaStream_t s;
  ~DevVecs() {
    cudaStreamSynchronize(s);
    for (auto x : p) cudaFree(x);
  }
  double* add(size_t n) {
    p.push_back((double*)sbdgpu::dev_alloc(sizeof(double) * n));
    return p.back();
  }
};

// swap of framework/dm_vector.h:89-101: X <- b Y, Y <- a X
__global__ void swap_kernel(double a, double* __restrict__ X, double b, double* __restrict__ Y, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double c = a * X[i];
    X[i] = b * Y[i];
    Y[i] = c;
  }
}

void lanczos(sbdgpu_genop* g, double* Wh, int max_it, double eps, double* energy, int* n_iter) {
  if (max_it < 1) throw Error{SBDGPU_ERR_ARG, "max_it must be positive"};
  const size_t n = g->n;
  cudaStream_t st = g->base.stream;
  sbdgpu_ctx* c = &g->base;
  DevVecs v{{}, st};
  double* W = v.add(n);
  double* C0 = v.add(n);
  double* C1 = v.add(n);
  SBD_CUDA(cudaMemcpyAsync(W, Wh, sizeof(double) * n, cudaMemcpyHostToDevice, st));
  SBD_CUDA(cudaMemcpyAsync(C0, W, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  SBD_CUDA(cudaMemsetAsync(C1, 0, sizeof(double) * n, st));
  const int lda = max_it;
  std::vector<double> A((size_t)lda * lda, 0.0), U((size_t)lda * lda, 0.0), E(lda, 0.0);
  double e_old = 1.0e8;
  int it_stop = 0, steps = 0;
  const unsigned nblk = std::min<size_t>(blocks_for(n), 148 * 8);
  for (int it = 0; it < max_it; it++) {
    steps++;
    const int ii = it + lda * it, ij = it + lda * (it + 1), ji = it + 1 + lda * it;
    mult(g, C0, C1);
    const double aii = sbdgpu::dot(c, C0, C1, n);
    A[ii] = aii;
    for (int i = 0; i < steps; i++)
      for (int j = 0; j < steps; j++) U[i + lda * j] = A[i + lda * j];
    sbdgpu::jacobi_eig(steps, U.data(), lda, E.data());
    if (std::abs(E[0] - e_old) < eps || it + 1 == max_it) {
      it_stop = it;
      break;
    }
    e_old = E[0];
    sbdgpu::axpy(C1, C0, -aii, n, st);
    const double b = std::sqrt(sbdgpu::dot(c, C1, C1, n));
    sbdgpu::scale(C1, 1.0 / b, n, st);
    A[ij] = A[ji] = b;
    if (std::abs(b) < eps) {
      it_stop = it;
      break;
    }
    swap_kernel<<<nblk, kThreads, 0, st>>>(-b, C0, 1.0, C1, n);
    SBD_CUDA(cudaGetLastError());
  }
  // the Ritz vector from a second pass of the recurrence (lanczos.h:276-302)
  SBD_CUDA(cudaMemcpyAsync(C0, W, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  SBD_CUDA(cudaMemsetAsync(C1, 0, sizeof(double) * n, st));
  sbdgpu::scale(W, U[0], n, st);
  for (int it = 0; it < it_stop; it++) {
    const int ii = it + lda * it;
    mult(g, C0, C1);
    sbdgpu::axpy(C1, C0, -A[ii], n, st);
    const double b = std::sqrt(sbdgpu::dot(c, C1, C1, n));
    sbdgpu::scale(C1, 1.0 / b, n, st);
    sbdgpu::axpy(W, C1, U[it + 1], n, st);
    swap_kernel<<<nblk, kThreads, 0, st>>>(-b, C0, 1.0, C1, n);
    SBD_CUDA(cudaGetLastError());
  }
  SBD_CUDA(cudaMemcpyAsync(Wh, W, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
  SBD_CUDA(cudaStreamSynchronize(st));
  if (energy) *energy = E[0];
  if (n_iter) *n_iter = steps;
}

void davidson(sbdgpu_genop* g, const sbdgpu_opts* o, double* Wh, double* energy, double* trace_e, double* trace_tol,
              int max_trace, int* n_steps) {
  const int nb = o->max_nb;
  if (nb < 1 || nb > 32) throw Error{SBDGPU_ERR_ARG, "max_nb must be in [1, 32]"};
  const size_t n = g->n;
  cudaStream_t st = g->base.stream;
  sbdgpu_ctx* c = &g->base;
  DevVecs v{{}, st};
  double* W = v.add(n);
  double* R = v.add(n);
  double* hii = v.add(n);
  std::vector<double*> C(nb), HC(nb);
  for (int k = 0; k < nb; k++) {
    C[k] = v.add(n);
    HC[k] = v.add(n);
  }
  diagonal(g, hii);
  SBD_CUDA(cudaMemcpyAsync(W, Wh, sizeof(double) * n, cudaMemcpyHostToDevice, st));
  const double eps_reg = 1.0e-12;
  std::vector<double> H(nb * nb, 0.0), U(nb * nb, 0.0), E(nb, 0.0);
  int steps = 0;
  bool cont = true;
  for (int it = 0; it < o->max_it && cont; it++) {
    SBD_CUDA(cudaMemcpyAsync(C[0], W, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    for (int ib = 0; ib < nb; ib++) {
      SBD_CUDA(cudaMemsetAsync(HC[ib], 0, sizeof(double) * n, st));
      mult(g, C[ib], HC[ib]);
      for (int jb = 0; jb <= ib; jb++) {
        H[jb + nb * ib] = sbdgpu::dot(c, C[jb], HC[ib], n);
        H[ib + nb * jb] = H[jb + nb * ib];
      }
      for (int jb = 0; jb <= ib; jb++)
        for (int kb = 0; kb <= ib; kb++) U[jb + nb * kb] = H[jb + nb * kb];
      sbdgpu::jacobi_eig(ib + 1, U.data(), nb, E.data());
      sbdgpu::ritz_update(C.data(), HC.data(), U.data(), ib + 1, E[0], W, R, n, st);
      const double nw = std::sqrt(sbdgpu::dot(c, W, W, n));
      sbdgpu::scale(W, 1.0 / nw, n, st);
      const double tol = std::sqrt(sbdgpu::dot(c, R, R, n));
      sbdgpu::scale(R, 1.0 / tol, n, st);
      if (trace_e && steps < max_trace) trace_e[steps] = E[0];
      if (trace_tol && steps < max_trace) trace_tol[steps] = tol;
      steps++;
      if (o->verbose) {
        std::cout << " Davidson iteration " << it << "." << ib << " (tol = " << tol << "):";
        for (int p = 0; p < std::min(ib + 1, 4); p++) std::cout << " " << E[p];
        std::cout << std::endl;
      }
      if (tol < o->eps) {
        cont = false;
        break;
      }
      if (ib < nb - 1) {
        sbdgpu::precondition(R, hii, E[0], eps_reg, C[ib + 1], n, st);
        for (int kb = 0; kb < ib + 1; kb++) {
          const double olap = sbdgpu::dot(c, C[kb], C[ib + 1], n);
          sbdgpu::axpy(C[ib + 1], C[kb], -olap, n, st);
        }
        const double nc = std::sqrt(sbdgpu::dot(c, C[ib + 1], C[ib + 1], n));
        sbdgpu::scale(C[ib + 1], 1.0 / nc, n, st);
      }
    }
  }
  SBD_CUDA(cudaMemsetAsync(R, 0, sizeof(double) * n, st));
  mult(g, W, R);
  const double e = sbdgpu::dot(c, W, R, n);
  SBD_CUDA(cudaMemcpyAsync(Wh, W, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
  SBD_CUDA(cudaStreamSynchronize(st));
  if (energy) *energy = e;
  if (n_steps) *n_steps = steps;
}


// ---------------------------------------------------------------- the expanded space
//
// MeasHamSquare and ExpandBasis (expand.h:10-366) look past the basis: every
// configuration an off-diagonal term reaches from a basis state, with weight
// coef * sign * W_i.  Here a count pass and a write pass (one warp per state
// over its applicable buckets, as in the mult) lay those out with the basis
// states themselves first, a radix sort (CUB) orders them by configuration,
// and head flags mark each distinct configuration.  One-word configurations
// are sorted themselves, with their weights where those are wanted, over the
// bits that occur; wider ones through their indices, least significant word
// first.  Every state testing every term in a thread of its own took 97 % of
// the GPU time of a 4,900-state expansion (21 ms a call).

constexpr int kGenThreads = 256;

// entries of state i: 1 (itself) + its applicable off-diagonal terms (with
// |coef sign W_i| > eps when select)
template <int NW>
__global__ void __launch_bounds__(kGenThreads) gen_count_kernel(const uint64_t* __restrict__ states, size_t n,
                                                               TermList<NW> tl, const double* __restrict__ W,
                                                               double eps, int select, int64_t* __restrict__ counts) {
  const int lane = threadIdx.x & 31;
  const size_t warps = ((size_t)gridDim.x * kGenThreads) >> 5;
  for (size_t i = ((size_t)blockIdx.x * kGenThreads + threadIdx.x) >> 5; i < n; i += warps) {
    uint64_t v[NW];
#pragma unroll
    for (int x = 0; x < NW; x++) v[x] = __ldg(&states[i * NW + x]);
    const double wi = W[i];
    int64_t cnt = 1;
    for_terms<NW>(tl, v, [&](bool on, const uint64_t (&)[NW], double c) {
      cnt += __popc(__ballot_sync(0xffffffffu, on && (!select || fabs(c * wi) > eps)));
    });
    if (lane == 0) counts[i] = cnt;
  }
}

template <int NW>
__global__ void __launch_bounds__(kGenThreads) gen_write_kernel(const uint64_t* __restrict__ states, size_t n,
                                                               TermList<NW> tl, const double* __restrict__ W,
                                                               const double* __restrict__ hdiag, double eps, int select,
                                                               const int64_t* __restrict__ offs,
                                                               uint64_t* __restrict__ keys, double* __restrict__ vals) {
  const int lane = threadIdx.x & 31;
  const size_t warps = ((size_t)gridDim.x * kGenThreads) >> 5;
  for (size_t i = ((size_t)blockIdx.x * kGenThreads + threadIdx.x) >> 5; i < n; i += warps) {
    uint64_t v[NW];
#pragma unroll
    for (int x = 0; x < NW; x++) v[x] = __ldg(&states[i * NW + x]);
    const double wi = W[i];
    int64_t o = offs[i];
    if (lane == 0) {
#pragma unroll
      for (int x = 0; x < NW; x++) keys[(size_t)o * NW + x] = v[x];
      if (vals) vals[o] = hdiag[i] * wi;  // the diagonal list's weight (expand.h:43-64)
    }
    o++;
    for_terms<NW>(tl, v, [&](bool on, const uint64_t (&w)[NW], double c) {
      const double val = c * wi;
      const bool put = on && (!select || fabs(val) > eps);
      const unsigned m = __ballot_sync(0xffffffffu, put);
      if (put) {
        const size_t at = (size_t)o + __popc(m & ((1u << lane) - 1u));
#pragma unroll
        for (int x = 0; x < NW; x++) keys[at * NW + x] = w[x];
        if (vals) vals[at] = val;
      }
      o += __popc(m);
    });
  }
}

__global__ void iota_kernel(int64_t* __restrict__ out, size_t m) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (size_t)gridDim.x * blockDim.x)
    out[i] = (int64_t)i;
}

// entry of sorted place i (idx null: the entries themselves are sorted)
__device__ __forceinline__ size_t entry(const int64_t* __restrict__ idx, size_t i) {
  return idx ? (size_t)idx[i] : i;
}

__global__ void gather_word_kernel(const uint64_t* __restrict__ keys, int nw, int word,
                                   const int64_t* __restrict__ idx, uint64_t* __restrict__ out, size_t m) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (size_t)gridDim.x * blockDim.x)
    out[i] = keys[(size_t)idx[i] * nw + word];
}

// head[i] = 1 where sorted entry i starts a new configuration
__global__ void head_kernel(const uint64_t* __restrict__ keys, int nw, const int64_t* __restrict__ idx,
                            int64_t* __restrict__ head, size_t m) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (size_t)gridDim.x * blockDim.x) {
    int64_t h = i == 0;
    if (i > 0)
      for (int x = 0; x < nw; x++) h |= keys[entry(idx, i) * nw + x] != keys[entry(idx, i - 1) * nw + x];
    head[i] = h;
  }
}

// sums[seg[i]] += vals of sorted entry i (seg = inclusive scan of head - 1)
__global__ void seg_sum_kernel(const int64_t* __restrict__ seg, const int64_t* __restrict__ idx,
                               const double* __restrict__ vals, double* __restrict__ sums, size_t m) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (size_t)gridDim.x * blockDim.x)
    atomicAdd(&sums[seg[i] - 1], vals[entry(idx, i)]);
}

// out[seg[i]-1] = key of entry i for the heads
__global__ void compact_kernel(const uint64_t* __restrict__ keys, int nw, const int64_t* __restrict__ idx,
                               const int64_t* __restrict__ head, const int64_t* __restrict__ seg,
                               uint64_t* __restrict__ out, size_t m) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (size_t)gridDim.x * blockDim.x)
    if (head[i])
      for (int x = 0; x < nw; x++) out[(size_t)(seg[i] - 1) * nw + x] = keys[entry(idx, i) * nw + x];
}

}  // namespace


namespace {

// The expanded space of W: sorted entries (by idx, or themselves where idx is
// null), their configuration keys, weights (null when not wanted), head flags
// and segment numbers (inclusive scan of the heads), all on the device.
struct Expanded {
  std::vector<void*> bufs;
  cudaStream_t s = nullptr;
  uint64_t* keys = nullptr;
  double* vals = nullptr;
  int64_t* idx = nullptr;
  int64_t* head = nullptr;
  int64_t* seg = nullptr;
  size_t m = 0, distinct = 0;
  void* alloc(size_t bytes) {
    bufs.push_back(sbdgpu::dev_alloc(std::max<size_t>(bytes, 16)));
    return bufs.back();
  }
  ~Expanded() {
    if (s) cudaStreamSynchronize(s);
    for (auto p : bufs) cudaFree(p);
  }
};

// Slices of one allocation, 256-byte aligned.
struct Slices {
  size_t total = 0;
  size_t add(size_t bytes) {
    const size_t at = total;
    total += (bytes + 255) / 256 * 256;
    return at;
  }
};

template <int NW>
void expand_nw(sbdgpu_genop* g, const double* dW, double eps, int select, bool weights, Expanded& x) {
  cudaStream_t st = g->base.stream;
  x.s = st;
  const size_t n = g->n;
  const unsigned nblk = (unsigned)std::min<size_t>((n * 32 + kGenThreads - 1) / kGenThreads, 148 * 64);
  const TermList<NW> tl = term_list<NW>(g);
  size_t tscan = 0;
  SBD_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tscan, (int64_t*)nullptr, (int64_t*)nullptr, n + 1, st));
  Slices a;
  const size_t at_counts = a.add(sizeof(int64_t) * (n + 1)), at_offs = a.add(sizeof(int64_t) * (n + 1)),
               at_tmp = a.add(tscan);
  char* first = (char*)x.alloc(a.total);
  int64_t* counts = (int64_t*)(first + at_counts);
  int64_t* offs = (int64_t*)(first + at_offs);
  SBD_CUDA(cudaMemsetAsync(counts + n, 0, sizeof(int64_t), st));
  gen_count_kernel<NW><<<nblk, kGenThreads, 0, st>>>(g->states, n, tl, dW, eps, select, counts);
  SBD_CUDA(cudaGetLastError());
  SBD_CUDA(cub::DeviceScan::ExclusiveSum(first + at_tmp, tscan, counts, offs, n + 1, st));
  int64_t m = 0;
  SBD_CUDA(cudaMemcpyAsync(&m, offs + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  SBD_CUDA(cudaStreamSynchronize(st));
  x.m = (size_t)m;
  // bits above the highest site in use are equal in every configuration
  int end_bit[NW];
  for (int w = 0; w < NW; w++) {
    const uint64_t any = g->site_or[w] | g->term_or[w];
    end_bit[w] = any ? 64 - __builtin_clzll(any) : 0;
  }
  size_t tsort = 0, tseg = 0;
  uint64_t* kn = nullptr;
  double* vn = nullptr;
  int64_t* in = nullptr;
  if (NW > 1)
    SBD_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tsort, kn, kn, in, in, x.m, 0, 64, st));
  else if (weights)
    SBD_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tsort, kn, kn, vn, vn, x.m, 0, 64, st));
  else
    SBD_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tsort, kn, kn, x.m, 0, 64, st));
  SBD_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tseg, in, in, x.m, st));
  // one allocation: keys, weights, the sort's second buffers, head flags, segment numbers and the libraries' scratch
  Slices b;
  const size_t at_keys = b.add(sizeof(uint64_t) * x.m * NW), at_vals = b.add(weights ? sizeof(double) * x.m : 0),
               at_k2 = b.add(sizeof(uint64_t) * x.m), at_v2 = b.add(NW > 1 || weights ? sizeof(double) * x.m : 0),
               at_k3 = b.add(NW > 1 ? sizeof(uint64_t) * x.m : 0), at_i3 = b.add(NW > 1 ? sizeof(int64_t) * x.m : 0),
               at_head = b.add(sizeof(int64_t) * x.m), at_seg = b.add(sizeof(int64_t) * x.m),
               at_t = b.add(std::max(tsort, tseg));
  char* p = (char*)x.alloc(b.total);
  x.keys = (uint64_t*)(p + at_keys);
  x.vals = weights ? (double*)(p + at_vals) : nullptr;
  x.head = (int64_t*)(p + at_head);
  x.seg = (int64_t*)(p + at_seg);
  gen_write_kernel<NW><<<nblk, kGenThreads, 0, st>>>(g->states, n, tl, dW, g->hdiag, eps, select, offs, x.keys,
                                                     x.vals);
  SBD_CUDA(cudaGetLastError());
  const unsigned gb = (unsigned)std::min<size_t>((x.m + 255) / 256 + 1, 148 * 8);
  if constexpr (NW == 1) {
    uint64_t* k2 = (uint64_t*)(p + at_k2);
    double* v2 = (double*)(p + at_v2);
    if (weights) {
      SBD_CUDA(cub::DeviceRadixSort::SortPairs(p + at_t, tsort, x.keys, k2, x.vals, v2, x.m, 0, end_bit[0], st));
      x.vals = v2;
    } else {
      SBD_CUDA(cub::DeviceRadixSort::SortKeys(p + at_t, tsort, x.keys, k2, x.m, 0, end_bit[0], st));
    }
    x.keys = k2;
  } else {
    uint64_t *ka = (uint64_t*)(p + at_k2), *kb = (uint64_t*)(p + at_k3);
    int64_t *ia = (int64_t*)(p + at_v2), *ib = (int64_t*)(p + at_i3);
    iota_kernel<<<gb, 256, 0, st>>>(ia, x.m);
    SBD_CUDA(cudaGetLastError());
    // least significant word first (each radix pass is stable)
    for (int w = 0; w < NW; w++) {
      if (end_bit[w] == 0) continue;
      gather_word_kernel<<<gb, 256, 0, st>>>(x.keys, NW, w, ia, ka, x.m);
      SBD_CUDA(cudaGetLastError());
      SBD_CUDA(cub::DeviceRadixSort::SortPairs(p + at_t, tsort, ka, kb, ia, ib, x.m, 0, end_bit[w], st));
      std::swap(ia, ib);
    }
    x.idx = ia;
  }
  head_kernel<<<gb, 256, 0, st>>>(x.keys, NW, x.idx, x.head, x.m);
  SBD_CUDA(cudaGetLastError());
  SBD_CUDA(cub::DeviceScan::InclusiveSum(p + at_t, tseg, x.head, x.seg, x.m, st));
  int64_t d = 0;
  SBD_CUDA(cudaMemcpyAsync(&d, x.seg + x.m - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  SBD_CUDA(cudaStreamSynchronize(st));
  x.distinct = (size_t)d;
}

void expand_space(sbdgpu_genop* g, const double* dW, double eps, int select, bool weights, Expanded& x) {
  if (!g->ready) throw Error{SBDGPU_ERR_STATE, "no operator: call sbdgpu_genop_set_terms first"};
  switch (g->nw) {
    case 1: expand_nw<1>(g, dW, eps, select, weights, x); break;
    case 2: expand_nw<2>(g, dW, eps, select, weights, x); break;
    default: expand_nw<4>(g, dW, eps, select, weights, x); break;
  }
}

}  // namespace

namespace sbdgpu {
void genop_set_error(sbdgpu_genop* g, const std::string& msg) { g->base.err = msg; }
}  // namespace sbdgpu

extern "C" {

int sbdgpu_genop_create(sbdgpu_genop** out, int device, int nwords, size_t nstates, const uint64_t* states,
                        int sign) {
  if (!out) return SBDGPU_ERR_ARG;
  *out = nullptr;
  auto* g = new (std::nothrow) sbdgpu_genop();
  if (!g) return SBDGPU_ERR_ALLOC;
  g->base.device = device;
  int rc = guarded(g, [&] {
    if (nwords != 1 && nwords != 2 && nwords != 4) throw Error{SBDGPU_ERR_ARG, "nwords must be 1, 2 or 4"};
    if (nstates == 0 || !states) throw Error{SBDGPU_ERR_ARG, "empty basis"};
    g->nw = nwords;
    g->n = nstates;
    g->sign = sign ? 1 : 0;
    SBD_CUDA(cudaStreamCreateWithFlags(&g->base.stream, cudaStreamNonBlocking));
    switch (nwords) {
      case 1: build_basis<1>(g, states); break;
      case 2: build_basis<2>(g, states); break;
      default: build_basis<4>(g, states); break;
    }
    SBD_CUDA(cudaStreamSynchronize(g->base.stream));
  });
  if (rc != SBDGPU_OK) {  // a bad argument, or no memory on the device
    sbdgpu_genop_destroy(g);
    return rc;
  }
  *out = g;
  return SBDGPU_OK;
}

int sbdgpu_genop_set_terms(sbdgpu_genop* g, size_t n_diag, const int64_t* diag_off, const int32_t* diag_ops,
                           const int32_t* diag_ndag, const double* diag_coef, size_t n_off, const int64_t* off_off,
                           const int32_t* off_ops, const int32_t* off_ndag, const double* off_coef) {
  return guarded(g, [&] {
    if ((n_diag && (!diag_off || !diag_ndag || !diag_coef)) || (n_off && (!off_off || !off_ndag || !off_coef)))
      throw Error{SBDGPU_ERR_ARG, "null term array"};
    switch (g->nw) {
      case 1:
        set_terms_nw<1>(g, n_diag, diag_off, diag_ops, diag_ndag, diag_coef, n_off, off_off, off_ops, off_ndag,
                        off_coef);
        break;
      case 2:
        set_terms_nw<2>(g, n_diag, diag_off, diag_ops, diag_ndag, diag_coef, n_off, off_off, off_ops, off_ndag,
                        off_coef);
        break;
      default:
        set_terms_nw<4>(g, n_diag, diag_off, diag_ops, diag_ndag, diag_coef, n_off, off_off, off_ops, off_ndag,
                        off_coef);
        break;
    }
  });
}

int sbdgpu_genop_mult_device(sbdgpu_genop* g, const double* dC, double* dW) {
  return guarded(g, [&] {
    if (!dC || !dW) throw Error{SBDGPU_ERR_ARG, "null vector"};
    mult(g, dC, dW);
    SBD_CUDA(cudaStreamSynchronize(g->base.stream));
  });
}

int sbdgpu_genop_mult(sbdgpu_genop* g, const double* C, double* W) {
  return guarded(g, [&] {
    if (!C || !W) throw Error{SBDGPU_ERR_ARG, "null vector"};
    cudaStream_t st = g->base.stream;
    DevVecs v{{}, st};
    double* dC = v.add(g->n);
    double* dW = v.add(g->n);
    SBD_CUDA(cudaMemcpyAsync(dC, C, sizeof(double) * g->n, cudaMemcpyHostToDevice, st));
    SBD_CUDA(cudaMemcpyAsync(dW, W, sizeof(double) * g->n, cudaMemcpyHostToDevice, st));
    mult(g, dC, dW);
    SBD_CUDA(cudaMemcpyAsync(W, dW, sizeof(double) * g->n, cudaMemcpyDeviceToHost, st));
    SBD_CUDA(cudaStreamSynchronize(st));
  });
}

int sbdgpu_genop_diagonal(sbdgpu_genop* g, double* hii) {
  return guarded(g, [&] {
    if (!hii) throw Error{SBDGPU_ERR_ARG, "null vector"};
    cudaStream_t st = g->base.stream;
    DevVecs v{{}, st};
    double* d = v.add(g->n);
    diagonal(g, d);
    SBD_CUDA(cudaMemcpyAsync(hii, d, sizeof(double) * g->n, cudaMemcpyDeviceToHost, st));
    SBD_CUDA(cudaStreamSynchronize(st));
  });
}

int sbdgpu_genop_lanczos(sbdgpu_genop* g, double* W, int max_it, double eps, double* energy, int* n_iter) {
  return guarded(g, [&] {
    if (!W) throw Error{SBDGPU_ERR_ARG, "null vector"};
    if (!g->ready) throw Error{SBDGPU_ERR_STATE, "no operator: call sbdgpu_genop_set_terms first"};
    lanczos(g, W, max_it, eps, energy, n_iter);
  });
}

int sbdgpu_genop_davidson(sbdgpu_genop* g, const sbdgpu_opts* opts, double* W, double* energy, double* trace_e,
                          double* trace_tol, int max_trace, int* n_steps) {
  return guarded(g, [&] {
    if (!opts || !W) throw Error{SBDGPU_ERR_ARG, "null argument"};
    if (!g->ready) throw Error{SBDGPU_ERR_STATE, "no operator: call sbdgpu_genop_set_terms first"};
    davidson(g, opts, W, energy, trace_e, trace_tol, max_trace, n_steps);
  });
}

int sbdgpu_genop_ham_square(sbdgpu_genop* g, const double* W, double* res) {
  return guarded(g, [&] {
    if (!W || !res) throw Error{SBDGPU_ERR_ARG, "null argument"};
    cudaStream_t st = g->base.stream;
    DevVecs v{{}, st};
    double* dW = v.add(g->n);
    SBD_CUDA(cudaMemcpyAsync(dW, W, sizeof(double) * g->n, cudaMemcpyHostToDevice, st));
    Expanded x;
    expand_space(g, dW, 0.0, 0, true, x);
    double* sums = v.add(x.distinct);
    SBD_CUDA(cudaMemsetAsync(sums, 0, sizeof(double) * x.distinct, st));
    const unsigned gb = (unsigned)std::min<size_t>((x.m + 255) / 256 + 1, 148 * 8);
    seg_sum_kernel<<<gb, 256, 0, st>>>(x.seg, x.idx, x.vals, sums, x.m);
    SBD_CUDA(cudaGetLastError());
    *res = sbdgpu::dot(&g->base, sums, sums, x.distinct);
  });
}

int sbdgpu_genop_expand(sbdgpu_genop* g, const double* W, double eps_hb, uint64_t* out, size_t capacity,
                        size_t* n_out) {
  return guarded(g, [&] {
    if (!W || !n_out) throw Error{SBDGPU_ERR_ARG, "null argument"};
    cudaStream_t st = g->base.stream;
    DevVecs v{{}, st};
    double* dW = v.add(g->n);
    SBD_CUDA(cudaMemcpyAsync(dW, W, sizeof(double) * g->n, cudaMemcpyHostToDevice, st));
    Expanded x;
    expand_space(g, dW, eps_hb, 1, false, x);
    *n_out = x.distinct;
    if (!out) return;
    if (capacity < x.distinct) throw Error{SBDGPU_ERR_LIMIT, "output holds fewer states than the expanded basis"};
    uint64_t* d = (uint64_t*)x.alloc(sizeof(uint64_t) * x.distinct * g->nw);
    const unsigned gb = (unsigned)std::min<size_t>((x.m + 255) / 256 + 1, 148 * 8);
    compact_kernel<<<gb, 256, 0, st>>>(x.keys, g->nw, x.idx, x.head, x.seg, d, x.m);
    SBD_CUDA(cudaGetLastError());
    SBD_CUDA(cudaMemcpyAsync(out, d, sizeof(uint64_t) * x.distinct * g->nw, cudaMemcpyDeviceToHost, st));
    SBD_CUDA(cudaStreamSynchronize(st));
  });
}

const char* sbdgpu_genop_last_error(sbdgpu_genop* g) { return g ? g->base.err.c_str() : "null object"; }

void sbdgpu_genop_destroy(sbdgpu_genop* g) {
  if (!g) return;
  cudaSetDevice(g->base.device);
  if (g->base.stream) cudaStreamSynchronize(g->base.stream);
  cudaFree(g->states);
  cudaFree(g->slots);
  cudaFree(g->slot_of);
  cudaFree(g->buckets);
  cudaFree(g->t_cre);
  cudaFree(g->t_sgn);
  cudaFree(g->t_coef);
  cudaFree(g->self_terms);
  cudaFree(g->hdiag);
  cudaFree(g->base.red);
  if (g->base.stream) cudaStreamDestroy(g->base.stream);
  g->base.red = nullptr;
  g->base.stream = nullptr;
  delete g;
}

}  // extern "C"
