// FRI compression of a dense FP64 tensor on the GPU, bit for bit equal to
// the reference's single-threaded fri_compression (fri-cc
// src/fri_utils.cpp:439-522, systematic sampling) and "largest" compression
// (include/sparse_tensor.hpp:46-56).
//
// Pipeline (x resident in HBM, N elements, keep m):
//   1. one pass over x: histogram of the top 12 bits of |x| and the chunk
//      sums of one_norm, then one_norm (:164-171) as an exact sequential
//      chain (exactsum.cuh);
//   2. a select digit: the elements at or above it hold every entry D can
//      take (k_select_digit), which is 0.2-2% of the m largest on MP2-like
//      amplitudes; their stable compaction (decoupled look-back, one pass)
//      and their sort by descending |x|, ties by ascending index: the order
//      of argsort(x, m) (:11-36), as far as it is needed;
//   3. the remaining-norm chain R -= |x_(d)| over the sorted candidates and
//      the acceptance test (m-d)|x_(d)| >= R-|x_(d)| && R > 1e-14
//      (:411-421), evaluated from exact chain values up to its first failure;
//   4. p_i = |x_i| / R * m' (:375, this operation order), the p > 1 check
//      (:383-395), the exact partial sums of p (:142-143) and, for every
//      interval [I_j, I_{j+1}), the samples u_k = k + rn that land in it
//      (:136, :147-157); unmatched samples keep index 0, as in the reference;
//   5. output D in sorted order then S ascending, values x_D and x_S/p_S.
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "exactsum.cuh"
#include "intdiv.cuh"
#include "radix.cuh"
#include "sparse.cuh"

namespace {

// The first select digit: the top `bits` bits of |x| below the sign, 12 by
// default (bits [62:51]: the exponent and one mantissa bit, half an octave
// per bin), 10-13 through FRICC_TUNE_SELECT_BITS.  A wider digit leaves
// fewer candidates for the sort; every width selects the same elements.
constexpr int DIG_BITS_DEFAULT = 12, DIG_BITS_MIN = 10, DIG_BITS_MAX = 13;
constexpr int NDIG = 1 << DIG_BITS_MAX;  // histogram words per compression

int select_bits() {
  const int b = fricc_tune_get(FRICC_TUNE_SELECT_BITS);
  return b >= DIG_BITS_MIN && b <= DIG_BITS_MAX ? b : DIG_BITS_DEFAULT;
}

__device__ __forceinline__ unsigned long long abs_key(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// Replica batches (R compressions of R equal-sized tensors in one set of
// launches): per-replica strides, in elements, of the n-sized arrays, the
// m-sized arrays and the tile-state words; `one` is 1 for single words and
// structs (0, with every stride 0, outside a batch).  The replica is
// blockIdx.y, or blockIdx.x for the one-block kernels.
struct Rep {
  int64_t n = 0, m = 0, tile = 0, one = 0;
};

// histogram of the first select digit (1 << bits bins of dynamic shared
// memory) and, with csum, the approximate sum of |x| over each exact::CH
// chunk, in one read of x (the one_norm chain's first pass).  Persistent
// blocks over chunks, so the bins are zeroed and flushed once per block.
__global__ void __launch_bounds__(256) k_hist_sums(const double* __restrict__ x, int64_t n, unsigned* __restrict__ hist,
                                                   int bits, double* __restrict__ csum, Rep rp = Rep{}) {
  const int64_t nch = fricc_cdiv(n, (int64_t)exact::CH);
  x += blockIdx.y * rp.n;
  hist += blockIdx.y * rp.one * NDIG;
  if (csum) csum += blockIdx.y * rp.one * (nch + 1);
  extern __shared__ unsigned h[];
  __shared__ double red[32];
  const int nb = 1 << bits, shift = 63 - bits;
  for (int i = threadIdx.x; i < nb; i += 256) h[i] = 0;
  __syncthreads();
  for (int64_t c = blockIdx.x; c < nch; c += gridDim.x) {
    const int64_t base = c * exact::CH;
    double v[exact::CH / 256];
#pragma unroll
    for (int r = 0; r < exact::CH / 256; ++r) {
      const int64_t i = base + r * 256 + threadIdx.x;
      v[r] = i < n ? x[i] : 0.0;
    }
    double acc = 0.0;
#pragma unroll
    for (int r = 0; r < exact::CH / 256; ++r) {
      const int64_t i = base + r * 256 + threadIdx.x;
      if (i < n) atomicAdd(&h[abs_key(v[r]) >> shift], 1u);
      acc += exact::abs_bits(v[r]);
    }
    if (csum) {
      const double tot = block_sum_det(acc, red);
      if (threadIdx.x == 0) csum[c] = tot;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += 256)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

// Values decided on the device between the phases of one compression.
struct Ctl {
  int64_t dmin;       // first select digit kept as a candidate
  int64_t ncand;      // candidates (every element at or above dmin)
  int64_t mchain;     // length of the remaining-norm chain: min(m, ncand)
  double norm;        // one_norm
  int64_t found;      // 1: |D| already found by the chain's first chunks (k_rem_first)
  int64_t nd;         // |D|
  int64_t mp;         // m - |D|
  unsigned long long dkey;  // |x| bits of the last element of D
  int64_t didx;       // its index (-1: D is empty)
  double R;           // remaining norm
  unsigned long long rv;  // recip_word(R)
  double mprime;      // (double)(m - |D|)
  int sample;         // 1: R > 0 and finite, so samples can land in intervals
  double rn;          // the uniform draw
  // pivotal sampling
  int64_t bad;        // the first segment of the parallel walk whose end is not the next one's start
  int64_t serial;     // 1: the walk has to be the serial one (k_piv_chain)
  int64_t jend;       // last element the sampler visits (it stops once m' indices are out)
  int64_t npush;      // indices emitted up to jend (chain), then in total (final)
  int64_t plast;      // the pivot after jend
  int broke;          // 1: the sampler stopped early with m' indices
};

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

constexpr unsigned long long ST_AGG = 1ull << 62, ST_INCL = 2ull << 62, ST_VAL = (1ull << 62) - 1;
constexpr long long SPIN_LIMIT = 1ll << 22;

// Stable compaction of {i : top digit of |x_i| >= dmin} into (ckey, cidx),
// in ascending i.  Tiles take tickets in launch order; each publishes its
// count and looks back over its predecessors for its output offset.
__global__ void __launch_bounds__(256) k_compact(const double* __restrict__ x, int64_t n, const Ctl* __restrict__ c,
                                                 unsigned long long* __restrict__ ckey, unsigned* __restrict__ cidx,
                                                 unsigned long long* tstate, unsigned* ticket, unsigned* err,
                                                 const unsigned long long* never_set, long long test_spins,
                                                 int shift, Rep rp = Rep{}) {
  constexpr int NT = 256, ITEMS = 16, TILE = NT * ITEMS;
  {
    const int64_t r = blockIdx.y;
    x += r * rp.n;
    c += r * rp.one;
    ckey += r * rp.n;
    cidx += r * rp.n;
    tstate += r * rp.tile;
    never_set += r * rp.tile;
    ticket += r * rp.one;
    err += r * rp.one;
  }
  const unsigned dmin = (unsigned)c->dmin;
  __shared__ int s_tile;
  __shared__ int64_t s_pre;
  __shared__ int64_t sm[33];
  if (threadIdx.x == 0) s_tile = (int)atomicAdd(ticket, 1u);
  __syncthreads();
  const int tile = s_tile;
  // a warp owns 512 consecutive elements, 32 per load (coalesced), and ranks
  // its keepers with ballots; one thread per 16 consecutive elements read
  // 128 bytes apart and took 148 us on 20 M elements
  const int64_t base = (int64_t)tile * TILE + (threadIdx.x >> 5) * (32 * ITEMS) + (threadIdx.x & 31);
  unsigned long long key[ITEMS];
  unsigned mask[ITEMS];
  int wtot = 0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int64_t i = base + 32 * k;
    key[k] = i < n ? abs_key(x[i]) : 0ull;
  }
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int64_t i = base + 32 * k;
    mask[k] = __ballot_sync(0xffffffffu, i < n && (unsigned)(key[k] >> shift) >= dmin);
    wtot += __popc(mask[k]);
  }
  int64_t tot;
  const int64_t excl_lane = block_excl_sum((threadIdx.x & 31) == 0 ? wtot : 0, sm, &tot);
  const int64_t excl = __shfl_sync(0xffffffffu, excl_lane, 0);
  if (threadIdx.x == 0) {
    int64_t pre = 0;
    if (tile == 0) {
      atomicExch(&tstate[0], ST_INCL | (unsigned long long)tot);
    } else {
      atomicExch(&tstate[tile], ST_AGG | (unsigned long long)tot);
      if (test_spins > 0 && tile == 1) {
        // test only: a bounded wait on a word nothing sets runs out
        long long w = 0;
        while (ld_acquire(never_set) == 0ull) {
          if (++w > test_spins) {
            atomicOr(err, FRICC_DEV_TIMEOUT);
            break;
          }
        }
      }
      int j = tile - 1;
      long long spins = 0;
      while (j >= 0) {
        const unsigned long long v = ld_acquire(&tstate[j]);
        const unsigned long long fl = v & ~ST_VAL;
        if (fl == 0) {
          if (++spins > SPIN_LIMIT) {
            atomicOr(err, FRICC_DEV_TIMEOUT);
            break;
          }
          continue;
        }
        pre += (int64_t)(v & ST_VAL);
        if (fl == ST_INCL) break;
        --j;
      }
      atomicExch(&tstate[tile], ST_INCL | (unsigned long long)(pre + tot));
    }
    s_pre = pre;
  }
  __syncthreads();
  int64_t o = s_pre + excl;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    if ((mask[k] >> (threadIdx.x & 31)) & 1u) {
      const int64_t at = o + __popc(mask[k] & ((1u << (threadIdx.x & 31)) - 1u));
      ckey[at] = key[k];
      cidx[at] = (unsigned)(base + 32 * k);
    }
    o += __popc(mask[k]);
  }
}

struct GenAbs {
  const double* x;
  int64_t rs = 0;  // replica stride of x
  __device__ __forceinline__ double operator()(int64_t i) const { return exact::abs_bits(x[i]); }
  __device__ __forceinline__ GenAbs at(int r) const { return GenAbs{x + r * rs, rs}; }
};

struct GenSorted {
  const unsigned long long* keys;
  int64_t rs = 0;
  __device__ __forceinline__ double operator()(int64_t i) const { return __longlong_as_double((long long)keys[i]); }
  __device__ __forceinline__ GenSorted at(int r) const { return GenSorted{keys + r * rs, rs}; }
};

// p_i of make_probability_vector (src/fri_utils.cpp:375,378-381); D membership
// is "at or before the last kept element in (|x| desc, index asc) order".
struct GenP {
  const double* x;
  const Ctl* c;
  int64_t rs = 0, cs = 0;  // replica strides of x and c
  __device__ __forceinline__ GenP at(int r) const { return GenP{x + r * rs, c + r * cs, rs, cs}; }
  __device__ __forceinline__ double operator()(int64_t i) const {
    const double a = exact::abs_bits(x[i]);
    const unsigned long long k = abs_key(a);
    const int64_t didx = c->didx;
    if (didx >= 0 && (k > c->dkey || (k == c->dkey && i <= didx))) return 0.0;
    const double p = __dmul_rn(div_by(a, c->R, c->rv), c->mprime);
    // with R <= 0 or not finite no sample can land anywhere: feed the exact
    // chain zeros (NaN addends would only slow it down), but keep any p > 1
    // visible to the check of make_probability_vector
    return (c->sample || p > 1.0) ? p : 0.0;
  }
  __device__ __forceinline__ double value(int64_t i) const {  // the reference's p_i itself
    const double a = exact::abs_bits(x[i]);
    const unsigned long long k = abs_key(a);
    const int64_t didx = c->didx;
    if (didx >= 0 && (k > c->dkey || (k == c->dkey && i <= didx))) return 0.0;
    return __dmul_rn(div_by(a, c->R, c->rv), c->mprime);
  }
};

// The probabilities once computed into P (one division per element instead
// of one per pass of the exact chain); the p > 1 check was made then.
struct GenPv {
  const double* P;
  const double* x;
  const Ctl* c;
  int64_t rs = 0, cs = 0;  // replica strides of P and x, and of c
  __device__ __forceinline__ GenPv at(int r) const { return GenPv{P + r * rs, x + r * rs, c + r * cs, rs, cs}; }
  __device__ __forceinline__ double operator()(int64_t i) const { return c->sample ? P[i] : 0.0; }
  __device__ __forceinline__ double value(int64_t i) const { return P[i]; }
};

// get_d_largest's acceptance test for the positions d of the sorted list;
// each thread keeps its first failure and a warp publishes one minimum (an
// atomic per failing position serialised ~2 M of them on one word: 1.28 ms).
struct ConsAccept {
  int64_t m;
  double* Rb;                    // [m+1]: R before element d; Rb[mchain]: after the last
  unsigned long long* first_fail;
  const Ctl* c;
  int64_t one = 0;               // 1 in a replica batch
  int64_t mchain = 0;
  unsigned long long mine = ~0ull;
  __device__ __forceinline__ ConsAccept at(int r) const {
    const Ctl* cr = c + r * one;
    return ConsAccept{m, Rb + r * one * (m + 1), first_fail + r * one, cr, one, cr->mchain};
  }
  __device__ __forceinline__ void operator()(int64_t d, double before, double after, double a) {
    Rb[d] = before;
    if (d == mchain - 1) Rb[mchain] = after;
    const bool acc = (__dmul_rn((double)(unsigned long long)(m - d), a) >= after) && (before > 1e-14);
    if (!acc && (unsigned long long)d < mine) mine = (unsigned long long)d;
  }
  __device__ __forceinline__ void finish() {
    const unsigned long long w = warp_min(mine);
    if (lane_id() == 0 && w != ~0ull) atomicMin(first_fail, w);
  }
};

// number of k in [0, mp) with fl(k + rn) < I  (u_k increases with k)
__device__ __noinline__ int64_t count_below(double I, double rn, int64_t mp) {
  if (!(I > rn)) return 0;
  double g = floor(I - rn);
  int64_t k = g < 0.0 ? 0 : (g > (double)mp ? mp : (int64_t)g);
  for (int it = 0; it < 64 && k > 0 && __dadd_rn((double)(k - 1), rn) >= I; ++it) --k;
  for (int it = 0; it < 64 && k < mp && __dadd_rn((double)k, rn) < I; ++it) ++k;
  return k;
}

// v in [0, 2^31) as floor(v 2^32), from its bits; false for anything else
__device__ __forceinline__ bool fix32(double v, long long& f) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const int e = (int)(u >> 52);  // the sign bit makes e >= 2048
  if (e >= 1023 + 31) return false;
  const unsigned long long M = (u & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
  const int sh = e - (1075 - 32);  // M 2^(e-1075) 2^32
  f = (long long)(sh >= 0 ? M << sh : (sh > -64 ? M >> -sh : 0ull));
  return true;
}

// sample_systematic's interval search: the samples of interval j.  The two
// counts come from 32-bit fixed point on the integer pipe (FP64 floor, add
// and compare per element made this pass FP64-bound, and a dependent chain
// of them ran for every item of a thread): with D = floor(I 2^32) -
// floor(rn 2^32) within 2^32 units of I - rn, a fraction of D at least 2^12
// units from an integer decides every k, since fl(k + rn) is off by at most
// 2^-23 (2^9 units) below 2^31; nearer ones (1 in 5e5) take count_below.
struct ConsSample {
  const Ctl* c;
  unsigned* S;
  int64_t cs = 0, ss = 0;  // replica strides of c and S
  double rn = 0.0;
  int64_t mp = 0;
  long long frn = 0;
  int ok = 0;  // 1: samples can land; 2: and rn has a fixed-point form
  __device__ __forceinline__ ConsSample at(int r) const {
    ConsSample q{c + r * cs, S + r * ss, cs, ss};
    q.rn = q.c->rn;
    q.mp = q.c->mp;
    q.ok = q.c->sample ? (fix32(q.rn, q.frn) && q.mp < (1ll << 31) ? 2 : 1) : 0;
    return q;
  }
  __device__ __forceinline__ int64_t count(double I) const {
    long long f;
    if (ok == 2 && fix32(I, f)) {
      const long long D = f - frn;
      const unsigned fr = (unsigned)D;
      if (fr - (1u << 12) <= 0xffffffffu - (1u << 13)) {
        const long long k = (D >> 32) + 1;
        return k < 0 ? 0 : (k > mp ? mp : k);
      }
    }
    return count_below(I, rn, mp);
  }
  // the next sample and where it lies, u_k = fl(k + rn) >= 0, as bits
  struct Run {
    int64_t k;
    long long u;
  };
  __device__ __forceinline__ bool runs() const { return ok == 2; }
  __device__ __forceinline__ long long place(int64_t k) const {
    return k < mp ? __double_as_longlong(__dadd_rn((double)k, rn)) : LLONG_MAX;
  }
  __device__ __forceinline__ Run start(double s) const {
    const int64_t k = count(s);
    return Run{k, place(k)};
  }
  __device__ __forceinline__ void step(Run& r, int64_t j, double s) const {
    while (r.u < __double_as_longlong(s)) {
      S[r.k] = (unsigned)j;
      r.u = place(++r.k);
    }
  }
  __device__ __forceinline__ void operator()(int64_t j, double lo, double hi, double p) const {
    const long long pb = __double_as_longlong(p);
    if (!ok || !(pb > 0 && pb <= 0x7ff0000000000000ll)) return;  // p > 0
    const int64_t k1 = count(hi);
    for (int64_t k = count(lo); k < k1; ++k) S[k] = (unsigned)j;
  }
};

// Two systematic samplers over one chain: the two compressions of the same
// tensor an iteration makes (different draws) share every phase up to the
// probabilities, and the partial sums too.
struct ConsSample2 {
  ConsSample a, b;
  __device__ __forceinline__ ConsSample2 at(int r) const { return ConsSample2{a.at(r), b.at(r)}; }
  struct Run {
    ConsSample::Run a, b;
  };
  __device__ __forceinline__ bool runs() const { return a.runs() && b.runs(); }
  __device__ __forceinline__ Run start(double s) const { return Run{a.start(s), b.start(s)}; }
  __device__ __forceinline__ void step(Run& r, int64_t j, double s) const {
    a.step(r.a, j, s);
    b.step(r.b, j, s);
  }
  __device__ __forceinline__ void operator()(int64_t j, double lo, double hi, double p) const {
    a(j, lo, hi, p);
    b(j, lo, hi, p);
  }
};

// The select digit (one block of 1024): the candidates are the elements at
// or above it.  For "largest" (c->norm unused, fri = 0) the largest digit d
// with count(digit >= d) >= m.  For FRI a higher one when the histogram
// already shows where get_d_largest must stop: with C elements at or above
// bin b, their sum at most S (counts times the bins' upper edges) and every
// other |x| below b's lower edge e, position C of the sorted list fails the
// acceptance test when (m - C) e < norm - S - e, so |D| <= C and only those C
// elements have to be sorted and chained.  (slack covers the chain's own
// rounding, at most C half-ulps of the norm, and that of S.)  A norm or a
// sum that is infinite or NaN keeps the m largest.  One thread walking the bins took
// 147 us; this takes ~6.
__global__ void __launch_bounds__(1024) k_select_digit(const unsigned* __restrict__ hist, int64_t m, Ctl* c, int bits,
                                                       int fri, Rep rp = Rep{}) {
  hist += blockIdx.x * rp.one * NDIG;
  c += blockIdx.x * rp.one;
  __shared__ int64_t sm[33];
  __shared__ double wsum[33];
  __shared__ int s_best;
  const int nb = 1 << bits, shift = 63 - bits, per = nb >> 10;  // bits >= 10
  // thread t owns the bins nb-1 - (t per + j), j < per: descending
  // (all bins loaded at once: one after another, a thread's loads took 5 us)
  constexpr int PER = NDIG >> 10;
  const int top = nb - 1 - (int)threadIdx.x * per;
  unsigned h[PER + 1];
#pragma unroll
  for (int j = 0; j <= PER; ++j) h[j] = j <= per && top - j >= 0 ? hist[top - j] : 0u;
  int64_t cnt = 0;
  double sum = 0.0;
#pragma unroll
  for (int j = 0; j < PER; ++j)
    if (j < per && h[j]) {
      cnt += h[j];
      sum += (double)h[j] * __longlong_as_double((long long)((unsigned long long)(top - j + 1) << shift));
    }
  int64_t tot;
  int64_t C = block_excl_sum(cnt, sm, &tot);
  double incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double w = __shfl_up_sync(0xffffffffu, incl, o);
    if ((int)lane_id() >= o) incl += w;
  }
  if (lane_id() == 31) wsum[warp_id()] = incl;
  if (threadIdx.x == 0) s_best = INT_MAX;
  __syncthreads();
  // the sums of the warps before this one, then of the lanes
  double S = (int)lane_id() < (int)warp_id() ? wsum[lane_id()] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
  {
    const double ex = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane_id() > 0) S += ex;
  }
  const double norm = fri ? c->norm : 0.0;
  const bool bound = fri && norm > 0.0 && norm < __longlong_as_double(0x7ff0000000000000ll);
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    if (j >= per) break;
    const int b = top - j;
    if (h[j]) S += (double)h[j] * __longlong_as_double((long long)((unsigned long long)(b + 1) << shift));
    C += h[j];
    bool stop = C >= m;
    // only where the next bin holds something can the bound improve
    if (!stop && bound && b > 0 && h[j + 1]) {
      const double e = __longlong_as_double((long long)((unsigned long long)b << shift));
      const double slack = norm * ((double)(C + 2) * 0x1p-52 + 0x1p-38);
      stop = (double)(m - C) * e < (norm - S - e - slack) * (1.0 - 0x1p-20);
    }
    if (stop) {
      atomicMin(&s_best, (int)threadIdx.x * per + j);
      break;
    }
  }
  __syncthreads();
  if (s_best != INT_MAX && s_best / per == (int)threadIdx.x) {
    c->dmin = nb - 1 - s_best;  // this thread's C stopped at that bin
    c->ncand = C;
    c->mchain = m < C ? m : C;
  }
  if (s_best == INT_MAX && threadIdx.x == 0) {  // fewer than m elements: not reached (m <= n)
    c->dmin = 0;
    c->ncand = tot;
    c->mchain = m < tot ? m : tot;
  }
}

// |D|, R, the D threshold and m' into the state of this compression.
__device__ __forceinline__ void set_d(Ctl* c, int64_t nd, double R, const unsigned long long* ckey,
                                      const unsigned* cidx, int64_t m) {
  c->nd = nd;
  c->mp = m - nd;
  c->rv = recip_word(R);
  c->mprime = (double)(unsigned long long)(m - nd);
  c->R = R;
  c->dkey = nd > 0 ? ckey[nd - 1] : 0ull;
  c->didx = nd > 0 ? (int64_t)cidx[nd - 1] : -1;
  c->sample = (c->R > 0.0 && isfinite(c->R)) ? 1 : 0;
}

// The first chunks of the remaining-norm chain, in one block, until the
// acceptance test first fails (D is usually a few thousand entries: one or
// two chunks).  Sets c->found, and the chain's general kernels then have
// nothing to do; a longer D leaves them the whole chain.  Up to this many chunks
// (m <= 32768) those kernels, ~15 us even with nothing to do, are not launched;
// a chunk takes ~4 us here, so a D that fills them costs no more than they did.
constexpr int REM_CHUNKS = 8;
__global__ void __launch_bounds__(1024) k_rem_first(ConsAccept ca0, const unsigned long long* ckey,
                                                    const unsigned* cidx, Ctl* c, Rep rp = Rep{}) {
  const int rep = blockIdx.x;
  ConsAccept ca = exact::replica_of(ca0, rep);
  ckey += rep * rp.n;
  cidx += rep * rp.n;
  c += rep * rp.one;
  __shared__ exact::ChunkSmem csm;
  __shared__ unsigned long long s_min[32];
  const GenSorted gen{ckey};
  const int64_t len = ca.mchain;
  double s = c->norm;
  if (len == 0) {  // no element can pass: D is empty
    if (threadIdx.x == 0) {
      set_d(c, 0, s, ckey, cidx, ca.m);
      c->found = 1;
    }
    return;
  }
  for (int64_t ch = 0; ch < REM_CHUNKS && ch * exact::CH < len; ++ch) {
    const int64_t base = ch * exact::CH;
    const int n_in = (int)(len - base < exact::CH ? len - base : exact::CH);
    s = exact::block_exact_chunk<1024, exact::CH / 1024>(gen, base, n_in, s, true, ca, csm);
    const unsigned long long f = block_min<unsigned long long>(ca.mine, s_min);
    const bool end = f == ~0ull && base + n_in == len;
    if (f != ~0ull || end) {
      const int64_t nd = end ? len : (int64_t)f;
      if (threadIdx.x == 0) {
        set_d(c, nd, ca.Rb[nd], ckey, cidx, ca.m);  // Rb[nd] was written before block_min's barriers
        c->found = 1;
      }
      return;
    }
  }
}

// After the general chain: |D|, R, the D threshold, m' (unless found before).
__global__ void k_finish_d(const unsigned long long* __restrict__ ffail, const double* __restrict__ Rb,
                           const unsigned long long* __restrict__ ckey, const unsigned* __restrict__ cidx, int64_t m,
                           Ctl* c, Ctl* c2, double rn2, const double* rn2_dev, int64_t rn_stride, Rep rp = Rep{}) {
  const int64_t r = blockIdx.x;
  c += r * rp.one;
  if (!c->found) {
    const int64_t nd = (int64_t)ffail[r * rp.one];
    const int64_t at = nd < c->mchain ? nd : c->mchain;
    set_d(c, at, Rb[r * rp.one * (m + 1) + at], ckey + r * rp.n, cidx + r * rp.n, m);
  }
  if (c2) {  // a paired compression's second state: the same, with its own draw
    c2 += r * rp.one;
    *c2 = *c;
    c2->rn = rn2_dev ? rn2_dev[r * rn_stride] : rn2;
  }
}

// Everything a compression needs zeroed or set, in one launch (six memsets,
// a copy and two fills before): one grid row per replica.
__global__ void k_init(unsigned* hist, unsigned long long* tstate, int64_t ntile1, unsigned* S, unsigned* S2,
                       int64_t m, Ctl* c, double rn, const double* rn_dev, int64_t rn_stride, unsigned* err,
                       unsigned* ticket, unsigned long long* ffail, double* dzero, unsigned* bar, double* psum,
                       int64_t nch1) {
  const int64_t r = blockIdx.y;
  hist += r * NDIG;
  tstate += r * ntile1;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = t0; i < NDIG; i += stride) hist[i] = 0;
  for (int64_t i = t0; i < ntile1; i += stride) tstate[i] = 0;
  if (S)
    for (int64_t i = t0; i < m; i += stride) S[r * m + i] = 0;
  if (S2)
    for (int64_t i = t0; i < m; i += stride) S2[r * m + i] = 0;
  for (int64_t i = t0; i < nch1; i += stride) psum[r * nch1 + i] = 0.0;
  if (t0 == 0) {
    Ctl z{};
    z.rn = rn_dev ? rn_dev[r * rn_stride] : rn;
    c[r] = z;
    err[r] = 0;
    ticket[r] = 0;
    ffail[r] = (unsigned long long)m;
    dzero[0] = 0.0;
    if (r == 0) bar[0] = 0;
  }
}

// D part of the output: flat = sorted index, value = x (src/fri_utils.cpp:494,498-500)
__global__ void k_out_d(const double* __restrict__ x, const unsigned* __restrict__ sidx, int64_t nd,
                        int64_t* __restrict__ flat, double* __restrict__ vals) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nd; i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned j = sidx[i];
    flat[i] = j;
    vals[i] = x[j];
  }
}

// The whole output: D in sorted order (flat = index, value = x), then S,
// flat = S_k, value = x / p (src/fri_utils.cpp:494-504); with meta, |D| and
// the error word of this compression.
template <class G>
__global__ void k_out(G gp0, int64_t n, const unsigned* __restrict__ sidx, const unsigned* __restrict__ S, int64_t m,
                      int64_t* __restrict__ flat, double* __restrict__ vals, const unsigned* err,
                      unsigned long long* meta, Rep rp = Rep{}) {
  const int64_t r = blockIdx.y;
  const G gp = exact::replica_of(gp0, r);
  sidx += r * rp.n;
  S += r * rp.m;
  flat += r * rp.m;
  vals += r * rp.m;
  const int64_t nd = gp.c->nd;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const bool d = i < nd;
    unsigned j = d ? sidx[i] : S[i - nd];
    if (j >= n) j = 0;  // only after a sort that gave up (its error bit is set): stay inside x
    flat[i] = j;
    vals[i] = d ? gp.x[j] : __ddiv_rn(gp.x[j], gp.value(j));
  }
  if (meta && blockIdx.x == 0 && threadIdx.x == 0) {
    meta[2 * r * rp.one] = (unsigned long long)nd;
    meta[2 * r * rp.one + 1] |= (unsigned long long)err[r * rp.one];
  }
}

__global__ void k_unpack(const int64_t* __restrict__ flat, int64_t m, int64_t d0, int64_t d1, int64_t d2, int64_t d3,
                         int* __restrict__ slots, unsigned* err, Rep rp = Rep{}) {
  flat += blockIdx.y * rp.m;
  slots += 4 * blockIdx.y * rp.m;
  err += 4 * blockIdx.y * rp.one;  // the low half of each status block's second word (16 bytes a replica)
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < m; s += (int64_t)gridDim.x * blockDim.x) {
    unsigned long long f = (unsigned long long)flat[s];
    const unsigned long long D1 = d1, D2 = d2, D3 = d3;
    if (f >= (unsigned long long)d0 * D1 * D2 * D3) {
      // an index a failed compression left behind: flagged, and unpacked as
      // (0,0,0,0) so that the contractions launched before the status is
      // read stay inside their operands
      atomicOr(err, FRICC_DEV_INDEX);
      f = 0;
    }
    const unsigned long long i0 = f / (D1 * D2 * D3);
    const unsigned long long i1 = f % (D1 * D2 * D3) / (D2 * D3);
    const unsigned long long i2 = f % (D2 * D3) / D3;
    const unsigned long long i3 = f % D3;
    slots[4 * s + 0] = (int)i0;
    slots[4 * s + 1] = (int)i1;
    slots[4 * s + 2] = (int)i2;
    slots[4 * s + 3] = (int)i3;
  }
}

// ---------------------------------------------------------------------------
// Pivotal sampling (src/fri_utils.cpp:63-127).  The sampler carries a weight
// a = p_0; for j = 1, 2, ...: a += p_j and one uniform rn_j is drawn; below 1
// the pivot i moves to j if rn_j < p_j / a; at or above 1, a -= 1 and one
// index is emitted: the pivot (which then moves to j) if
// rn_j < (1 - p_j) / (1 - a), else j; it stops once m' indices are out.
//
// Only the carried weight is a true recurrence (sequential FP64 with a
// wrap), and it does not depend on the draws, nor does which elements emit.
// So: (1) the weight is walked, in parallel segments (below), recording a_j
// and the wrap flag of every element, which fixes where the sampler stops and
// how many draws it consumes; (2) the draws arrive; (3) every decision is independent given
// a_j, p_j and rn_j; (4) the pivot an element emits is the last "take"
// before it, a max-scan; its slot in S is the count of emits before it, a
// sum-scan.  Per-element codes: bit 0 the pivot moves here, bit 1 the
// element emits, bit 2 it emits the pivot.
constexpr unsigned char PV_TAKE = 1, PV_EMIT = 2, PV_PIVOT = 4;

// P = the p vector, with the p > 1 check and (psum, zeroed beforehand) the
// approximate sum of each exact::CH chunk of the addends its chain takes.
// Four blocks share a chunk, so that a small tensor's spread over the chip.  The
// divisions by R run on the integer pipe (div_by): 20 M elements 503 -> 144 us,
// of which the FP64 multiplication and sum are 70.
constexpr int PV_SUB = 4;
__global__ void __launch_bounds__(256) k_pvec(GenP gp0, int64_t n, double* __restrict__ P, unsigned* err,
                                              double* __restrict__ psum, Rep rp = Rep{}) {
  constexpr int SUB = exact::CH / PV_SUB;
  const GenP gp = gp0.at(blockIdx.y);
  P += blockIdx.y * rp.n;
  err += blockIdx.y * rp.one;
  __shared__ double red[32];
  const int64_t base = (int64_t)blockIdx.x * SUB;
  bool bad = false;
  double acc = 0.0;
#pragma unroll
  for (int r = 0; r < SUB / 256; ++r) {
    const int64_t i = base + r * 256 + threadIdx.x;
    if (i < n) {
      const double p = gp.value(i);
      P[i] = p;
      // p > 1, by its bits (a comparison is an FP64 instruction)
      const long long u = __double_as_longlong(p);
      bad |= u > 0x3ff0000000000000ll && u <= 0x7ff0000000000000ll;
      acc += p;
    }
  }
  if (bad) atomicOr(err, FRICC_DEV_P_GT_ONE);
  if (psum && gp.c->sample) {  // R <= 0 or not finite: the chain runs over zeros (GenPv)
    const double tot = block_sum_det(acc, red);
    const int64_t nch1 = fricc_cdiv(n, (int64_t)exact::CH) + 1;
    // (the order of these four additions moves only the chain's prediction)
    if (threadIdx.x == 0) atomicAdd(&psum[blockIdx.y * rp.one * nch1 + blockIdx.x / PV_SUB], tot);
  }
}

// The weight walk in parallel.  After a wrap the weight is a multiple of
// 2^-52 (a sum in [1, 2) minus 1, exactly), and every later step rounds at
// 2^-53 or finer until the sum passes 1 again: two walks whose weights differ
// by a multiple d of 2^-52 round alike and stay d apart, as long as no sum of
// theirs falls on different sides of a power of two, except that a tie at the
// wrap itself (ulp 2^-52) goes by the parity of d.  Over a segment from one
// wrap to another the walk is therefore a map n -> n + (n odd ? d1 : d0) on
// n = a 2^52 near a predicted n, and such maps compose.
//
// The tensor is cut into regions of S elements; a segment starts at the
// first wrap of its region that the exact fixed-point prefix sums (mod 1, in
// 2^-64) predict (k_piv_starts).  k_piv_walk<1> walks every segment from its
// predicted start, once per parity, and leaves its map; k_piv_claims composes
// them to the start of each segment; k_piv_walk<2> walks each segment again from
// there with the sampler's own FP64 operations, writes a_j and the flags, and
// compares its end with the next segment's start.  If they all agree the
// recurrence holds from end to end: the result does not rest on the argument
// above.  Where one does not (a prediction within ~1e-12 of a power of
// two), the claims behind it are recomputed from its true end, twice; what
// then remains (and p outside [0, 1], m' = 0, a stretch without a wrap through
// half the tensor) is left to the serial walk.
//
// Bound by the latency of two dependent FP64 additions per element over one
// segment (~70 ns each): o13v57 (549,081 elements) 73 ms serial, 60 us so.
constexpr int PW_MIN = 128;          // elements per region, at least
constexpr int64_t PW_SEGS = 32768;   // regions, at most
constexpr double PW_ULP = 0x1p-52;

struct PivSegs {
  int64_t n, S, nseg;
  unsigned long long* f;    // sums of floor(p 2^64) per region, then exclusive prefixes
  int64_t* start;           // the segment's first element (a wrap), -1: none
  exact::Map* map;
  double* claim;            // the weight after element start
  double* end;              // the weight at the end of the segment
  int* cnt;                 // its wraps
};

__device__ __forceinline__ unsigned long long frac64(double p) {  // floor(p 2^64) mod 2^64, p in [0, 1]
  const unsigned long long u = (unsigned long long)__double_as_longlong(p);
  const int e = (int)(u >> 52);
  const unsigned long long m = (u & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
  const int sh = e - (1075 - 64);
  return sh >= 64 || sh <= -64 ? 0ull : (sh >= 0 ? m << sh : m >> -sh);
}

// region sums (one warp each) and the check of p
__global__ void __launch_bounds__(256) k_piv_sums(const double* __restrict__ P, PivSegs g, Ctl* c) {
  const int lane = threadIdx.x & 31;
  for (int64_t s = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); s < g.nseg; s += (int64_t)gridDim.x * 8) {
    const int64_t j1 = (s + 1) * g.S < g.n ? (s + 1) * g.S : g.n;
    unsigned long long f = 0;
    bool odd = false;
    for (int64_t j = s * g.S + lane; j < j1; j += 32) {
      const double p = P[j];
      f += frac64(p);
      odd |= (unsigned long long)__double_as_longlong(p) > 0x3ff0000000000000ull;  // not in [0, 1] (or -0, NaN)
    }
    f = warp_sum(f);
    if (__any_sync(0xffffffffu, odd) && lane == 0) c->serial = 1;
    if (lane == 0) g.f[s] = f;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    c->bad = g.nseg;
    if (c->mp == 0) c->serial = 1;
  }
}

// exclusive prefixes of the region sums (one block)
__global__ void __launch_bounds__(1024) k_piv_prefix(PivSegs g, const Ctl* c) {
  if (c->serial) return;
  __shared__ int64_t sm[33];
  int64_t run = 0;
  for (int64_t b = 0; b < g.nseg; b += 1024) {
    const int64_t s = b + threadIdx.x;
    const int64_t v = s < g.nseg ? (int64_t)g.f[s] : 0;
    int64_t tot;
    const int64_t ex = block_excl_sum(v, sm, &tot);  // wraps mod 2^64, as wanted
    if (s < g.nseg) g.f[s] = (unsigned long long)(run + ex);
    run += tot;
  }
}

__device__ __forceinline__ bool ge_one(double s) { return (__double_as_longlong(s) >> 32) >= 0x3ff00000ll; }

// one step of the sampler's weight
__device__ __forceinline__ bool piv_step(double& a, double p) {
  const double sum = __dadd_rn(a, p);
  const bool w = ge_one(sum);
  a = __dadd_rn(sum, w ? -1.0 : 0.0);  // (sum >= +0: adding 0 leaves it)
  return w;
}

// The segments' starts, one thread each: the first wrap of the region that the
// prefix sums predict, and the weight they predict after it.
__global__ void __launch_bounds__(64) k_piv_starts(const double* __restrict__ P, PivSegs g, const Ctl* c) {
  if (c->serial) return;
  const int64_t s = (int64_t)blockIdx.x * 64 + threadIdx.x;
  if (s >= g.nseg) return;
  if (s == 0) {
    g.start[0] = 0;
    return;
  }
  const int64_t j0 = s * g.S, j1 = j0 + g.S < g.n ? j0 + g.S : g.n;
  unsigned long long F = g.f[s];
  int64_t at = -1;
  constexpr int U = 8;  // elements loaded at once
  for (int64_t j = j0; j < j1 && at < 0; j += U) {
    double p[U];
#pragma unroll
    for (int q = 0; q < U; ++q) p[q] = j + q < j1 ? P[j + q] : 0.0;
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const unsigned long long F1 = F + frac64(p[q]);
      if (at < 0) {
        if (F1 < F) at = j + q;
        F = F1;
      }
    }
  }
  g.start[s] = at;
  if (at >= 0) g.claim[s] = (double)(long long)(F >> 12) * PW_ULP;
}

// One thread per segment.  PASS 1: walk both parities of the predicted weight to
// the next segment's start, leave the map (segment 0: its true end).  PASS 2: walk
// from the claimed weight, write a_j, the wrap flags and their number, and report
// an end that is not the next claim.
//
// Both passes together take ~280 ns per element of the longest segment, the
// serial walk ~136 per element of the tensor: a stretch without a wrap of more
// than 15/32 of it (one or two samples; a long run of zeros) leaves the whole walk
// to the serial one.  (549,081 elements, 1 sample: 155 ms, now 75; 3 samples, in
// parallel: 52.)
template <int PASS>
__global__ void __launch_bounds__(64) k_piv_walk(const double* __restrict__ P, PivSegs g, Ctl* c,
                                                 double* __restrict__ A, unsigned char* __restrict__ code,
                                                 int64_t from_bad) {
  if (c->serial) return;
  const int64_t s = (int64_t)blockIdx.x * 64 + threadIdx.x;
  if (s >= g.nseg) return;
  // a later round walks only what follows the segment that failed
  if (PASS == 2 && from_bad) {
    const int64_t first = from_bad == 1 ? g.cnt[g.nseg] : g.cnt[g.nseg + 1];  // the last round's bad segment
    if (first >= g.nseg || s <= first) return;
  }
  const int64_t at = g.start[s];
  if (at < 0) {
    if (PASS == 1) g.map[s] = exact::map_id();
    return;
  }
  // to the next segment's start
  int64_t last = g.n - 1, nxt = g.nseg;
  for (int64_t t = s + 1; t < g.nseg; ++t)
    if (g.start[t] >= 0) {
      last = g.start[t];
      nxt = t;
      break;
    }
  double a0, a1 = 0.0;
  if (PASS == 1) {
    if ((last - at) * 32 > g.n * 15) {
      c->serial = 1;
      return;
    }
    const long long n = s == 0 ? 0 : (long long)(g.claim[s] * 0x1p52);
    a0 = s == 0 ? P[0] : (double)(n & ~1ll) * PW_ULP;
    a1 = (double)(n | 1ll) * PW_ULP;
  } else {
    a0 = s == 0 ? P[0] : g.claim[s];
    if (s == 0) {
      A[0] = a0;
      code[0] = 0;
    }
  }
  const double b0 = a0, b1 = a1;
  int cnt = 0;
  bool w0 = false, w1 = false;
  constexpr int U = 8;  // elements loaded ahead
  double buf[U];
  int64_t j = at + 1;
#pragma unroll
  for (int q = 0; q < U; ++q) buf[q] = j + q <= last ? P[j + q] : 0.0;
  while (j <= last) {
    // (another segment may have left the walk to the serial one; asked inside the
    // inner loop, it cost 7% of the walk)
    if (PASS == 1 && *(volatile int64_t*)&c->serial) return;
    const int64_t stop = j + 128 * U <= last ? j + 128 * U : last + 1;
    for (; j < stop; j += U) {
      double cur[U];
#pragma unroll
      for (int q = 0; q < U; ++q) cur[q] = buf[q];
#pragma unroll
      for (int q = 0; q < U; ++q) buf[q] = j + U + q <= last ? P[j + U + q] : 0.0;
#pragma unroll
      for (int q = 0; q < U; ++q) {
        if (j + q <= last) {
          w0 = piv_step(a0, cur[q]);
          if (PASS == 1) {
            w1 = piv_step(a1, cur[q]);
          } else {
            A[j + q] = a0;
            code[j + q] = w0 ? PV_EMIT : 0;
            cnt += w0 ? 1 : 0;
          }
        }
      }
    }
  }
  if (PASS == 1) {
    if (s == 0) {
      g.end[0] = a0;
    } else {
      // (an end that is no wrap has no map: its claim will not hold)
      const bool ok = w0 && w1;
      g.map[s] = ok ? exact::Map{(int64_t)((a0 - b0) * 0x1p52), (int64_t)((a1 - b1) * 0x1p52)} : exact::map_id();
    }
  } else {
    g.end[s] = a0;
    g.cnt[s] = cnt;
    if (nxt < g.nseg && __double_as_longlong(g.claim[nxt]) != __double_as_longlong(a0))
      atomicMin(reinterpret_cast<unsigned long long*>(&c->bad), (unsigned long long)s);
  }
}

// The weights at the segments' starts (one block): the maps composed from
// the end of segment 0, or (a later round) from the true end of the segment
// that failed, whose number moves to cnt[nseg] (cnt[nseg + 1]).
__global__ void __launch_bounds__(1024) k_piv_claims(PivSegs g, Ctl* c, int round) {
  if (c->serial) return;
  __shared__ exact::Map smaps[33];
  const int64_t bad = c->bad;
  __syncthreads();
  if (round > 0) {
    if (threadIdx.x == 0) g.cnt[g.nseg + round - 1] = (int)bad;
    if (bad >= g.nseg) return;
    if (threadIdx.x == 0) c->bad = g.nseg;
  }
  const int64_t s0 = round > 0 ? bad + 1 : 1;
  const double a = round > 0 ? g.end[bad] : g.end[0];
  int64_t first = s0;  // the next live segment
  while (first < g.nseg && g.start[first] < 0) ++first;
  int64_t n = (int64_t)(a * 0x1p52);
  for (int64_t b = s0; b < g.nseg; b += 1024) {
    const int64_t s = b + threadIdx.x;
    const bool live = s < g.nseg && g.start[s] >= 0;
    exact::Map tot;
    const exact::Map pre = exact::block_excl_scan_map<1024>(live ? g.map[s] : exact::map_id(), smaps, &tot);
    // (the segment behind one that failed takes the weight itself, on or off the 2^-52 grid)
    if (live) g.claim[s] = s == first ? a : (double)exact::apply(pre, n) * PW_ULP;
    n = exact::apply(tot, n);
  }
}

// Where the sampler stops: the element of the m'-th wrap (one block).
__global__ void __launch_bounds__(1024) k_piv_end(PivSegs g, const unsigned char* __restrict__ code, Ctl* c) {
  if (c->serial) return;
  if (c->bad < g.nseg) {  // not proven after the last round
    if (threadIdx.x == 0) c->serial = 1;
    return;
  }
  __shared__ int64_t sm[33];
  __shared__ int64_t s_seg, s_left;
  if (threadIdx.x == 0) s_seg = -1;
  __syncthreads();
  const int64_t mp = c->mp;
  int64_t run = 0;
  for (int64_t b = 0; b < g.nseg; b += 1024) {
    const int64_t s = b + threadIdx.x;
    const int64_t k = s < g.nseg && g.start[s] >= 0 ? g.cnt[s] : 0;
    int64_t tot;
    const int64_t ex = run + block_excl_sum(k, sm, &tot);
    if (k > 0 && ex < mp && ex + k >= mp) {
      s_seg = s;
      s_left = mp - ex;
    }
    run += tot;
  }
  __syncthreads();
  if (s_seg < 0) {
    if (threadIdx.x == 0) {
      c->jend = g.n - 1;
      c->npush = run;
      c->broke = 0;
    }
    return;
  }
  if (threadIdx.x < 32) {  // the left-th wrap of that segment
    int64_t left = s_left;
    for (int64_t j0 = g.start[s_seg] + 1;; j0 += 32) {
      const int64_t j = j0 + threadIdx.x;
      const unsigned w = __ballot_sync(0xffffffffu, j < g.n && code[j] != 0);
      if (__popc(w) >= left) {
        unsigned m = w;
        for (int64_t q = 1; q < left; ++q) m &= m - 1;
        if (threadIdx.x == 0) {
          c->jend = j0 + __ffs((int)m) - 1;
          c->npush = mp;
          c->broke = 1;
        }
        break;
      }
      left -= __popc(w);
      if (j0 + 32 >= g.n) break;  // not reached: the wraps were counted
    }
  }
}

// The serial walk, for what the parallel one leaves (c->serial).  One warp.
// Lane t of a batch of 32 elements keeps a_j and the wrap flag
// of element j0 + t; every lane walks the same chain (the p_j come in by
// shuffle, the next batch's are loaded while this one runs).
__global__ void __launch_bounds__(32) k_piv_chain(const double* __restrict__ P, int64_t n, Ctl* c,
                                                  double* __restrict__ A, unsigned char* __restrict__ code) {
  if (!c->serial) return;
  const int lane = threadIdx.x;
  const int64_t mp = c->mp;
  double a = P[0];
  if (lane == 0) {
    A[0] = a;
    code[0] = 0;
  }
  int64_t cnt = 0, jend = n - 1;
  int broke = 0;
  double pn = 1 + lane < n ? P[1 + lane] : 0.0;
  for (int64_t j0 = 1; j0 < n; j0 += 32) {
    const double pj = pn;
    const int64_t jn = j0 + 32 + lane;
    pn = jn < n ? P[jn] : 0.0;
    double myA = 0.0;
    bool myW = false;
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const double pt = __shfl_sync(0xffffffffu, pj, t);
      const double sum = __dadd_rn(a, pt);
      const bool w = !(sum < 1.0);
      a = w ? __dsub_rn(sum, 1.0) : sum;
      if (lane == t) {
        myA = a;
        myW = w;
      }
    }
    const int64_t j = j0 + lane;
    const bool valid = j < n;
    const unsigned wm = __ballot_sync(0xffffffffu, myW && valid);
    // the first element of this batch after which exactly m' indices are out
    int stop = -1;
    if (mp == 0) {
      if (j0 == 1 && !(wm & 1u)) stop = 0;
    } else if (cnt < mp && cnt + __popc(wm) >= mp) {
      int64_t r = mp - cnt;
      for (int b = 0; b < 32; ++b)
        if (((wm >> b) & 1u) && --r == 0) {
          stop = b;
          break;
        }
    }
    if (valid && (stop < 0 || lane <= stop)) {
      A[j] = myA;
      code[j] = myW ? PV_EMIT : 0;
    }
    if (stop >= 0) {
      jend = j0 + stop;
      broke = 1;
      cnt = mp;
      break;
    }
    cnt += __popc(wm);
  }
  if (lane == 0) {
    c->jend = jend;
    c->npush = cnt;
    c->broke = broke;
  }
}

// decisions for j in [1, jend], with rn_j = R[j-1]
__global__ void k_piv_decide(const double* __restrict__ P, const double* __restrict__ A,
                             unsigned char* __restrict__ code, const double* __restrict__ R, const Ctl* c,
                             unsigned* err) {
  const int64_t jend = c->jend;
  bool bad = false;
  for (int64_t j = 1 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j <= jend;
       j += (int64_t)gridDim.x * blockDim.x) {
    const double rn = R[j - 1], p = P[j], a = A[j];
    unsigned char cd = code[j];
    if (!(cd & PV_EMIT)) {
      if (rn < __ddiv_rn(p, a)) cd |= PV_TAKE;
    } else {
      const double pa = __ddiv_rn(__dsub_rn(1.0, p), __dsub_rn(1.0, a));
      bad |= pa > 1.0 || pa < 0.0;
      if (rn < pa) cd |= PV_TAKE | PV_PIVOT;
    }
    code[j] = cd;
  }
  if (bad) atomicOr(err, FRICC_DEV_PIVOTAL);
}

constexpr int PV_NT = 256, PV_IT = 16, PV_TILE = PV_NT * PV_IT;

// block-wide exclusive max of int64 (identity -1), thread order; smem >= 33
__device__ __forceinline__ int64_t block_excl_max(int64_t v, int64_t* smem, int64_t* total) {
  int64_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t w = __shfl_up_sync(0xffffffffu, incl, o);
    if ((int)lane_id() >= o && w > incl) incl = w;
  }
  const int64_t excl_w = __shfl_up_sync(0xffffffffu, incl, 1);
  const int nw = blockDim.x >> 5;
  __syncthreads();
  if (lane_id() == 31) smem[warp_id()] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int64_t run = -1;
    for (int w = 0; w < nw; ++w) {
      const int64_t t = smem[w];
      smem[w] = run;
      run = t > run ? t : run;
    }
    smem[32] = run;
  }
  __syncthreads();
  int64_t r = smem[warp_id()];
  if (lane_id() > 0 && excl_w > r) r = excl_w;
  *total = smem[32];
  __syncthreads();
  return r;
}

// per tile: the last take and the number of emits among j in [1, jend]
__global__ void __launch_bounds__(PV_NT) k_piv_tiles(const unsigned char* __restrict__ code, const Ctl* c,
                                                     int64_t* __restrict__ tlast, int64_t* __restrict__ tcnt) {
  __shared__ int64_t sm[33];
  const int64_t jend = c->jend;
  const int64_t j0 = (int64_t)blockIdx.x * PV_TILE + (int64_t)threadIdx.x * PV_IT;
  int64_t last = -1, cnt = 0;
#pragma unroll
  for (int k = 0; k < PV_IT; ++k) {
    const int64_t j = j0 + k;
    if (j >= 1 && j <= jend) {
      const unsigned char cd = code[j];
      if (cd & PV_TAKE) last = j;
      cnt += (cd & PV_EMIT) ? 1 : 0;
    }
  }
  int64_t tot_last, tot_cnt;
  block_excl_max(last, sm, &tot_last);
  block_excl_sum(cnt, sm, &tot_cnt);
  if (threadIdx.x == 0) {
    tlast[blockIdx.x] = tot_last;
    tcnt[blockIdx.x] = tot_cnt;
  }
}

// exclusive scans over tiles, in place; the pivot starts at index 0
__global__ void __launch_bounds__(1024) k_piv_carry(int64_t* __restrict__ tlast, int64_t* __restrict__ tcnt,
                                                    int64_t ntile, Ctl* c) {
  __shared__ int64_t sm[33];
  int64_t run_last = 0, run_cnt = 0;
  for (int64_t b = 0; b < ntile; b += 1024) {
    const int64_t t = b + threadIdx.x;
    const int64_t l = t < ntile ? tlast[t] : -1, k = t < ntile ? tcnt[t] : 0;
    int64_t tl, tk;
    int64_t el = block_excl_max(l, sm, &tl);
    const int64_t ek = block_excl_sum(k, sm, &tk);
    el = el > run_last ? el : run_last;
    if (t < ntile) {
      tlast[t] = el;
      tcnt[t] = run_cnt + ek;
    }
    run_last = tl > run_last ? tl : run_last;
    run_cnt += tk;
  }
  if (threadIdx.x == 0) {
    c->plast = run_last;
    c->npush = run_cnt;
  }
}

// S[slot] for every emit with slot < m'
__global__ void __launch_bounds__(PV_NT) k_piv_emit(const unsigned char* __restrict__ code,
                                                    const int64_t* __restrict__ clast,
                                                    const int64_t* __restrict__ ccnt, const Ctl* c,
                                                    unsigned* __restrict__ S) {
  __shared__ int64_t sm[33];
  const int64_t jend = c->jend, mp = c->mp;
  const int64_t j0 = (int64_t)blockIdx.x * PV_TILE + (int64_t)threadIdx.x * PV_IT;
  unsigned char cd[PV_IT];
  int64_t last = -1, cnt = 0;
#pragma unroll
  for (int k = 0; k < PV_IT; ++k) {
    const int64_t j = j0 + k;
    cd[k] = (j >= 1 && j <= jend) ? code[j] : 0;
    if (cd[k] & PV_TAKE) last = j;
    cnt += (cd[k] & PV_EMIT) ? 1 : 0;
  }
  int64_t tl, tk;
  int64_t piv = block_excl_max(last, sm, &tl);
  int64_t slot = block_excl_sum(cnt, sm, &tk);
  const int64_t cl = clast[blockIdx.x];
  piv = piv > cl ? piv : cl;
  slot += ccnt[blockIdx.x];
#pragma unroll
  for (int k = 0; k < PV_IT; ++k) {
    const int64_t j = j0 + k;
    if (cd[k] & PV_EMIT) {
      if (slot < mp) S[slot] = (unsigned)((cd[k] & PV_PIVOT) ? piv : j);
      ++slot;
    }
    if (cd[k] & PV_TAKE) piv = j;
  }
}

// the end of the walk: a sampler that visited every element emits its pivot
// when |a - 1| < 1e-5; the count must come out at m'
__global__ void k_piv_final(const double* __restrict__ A, int64_t n, Ctl* c, unsigned* __restrict__ S,
                            unsigned* err) {
  int64_t np = c->npush;
  bool bad = false;
  if (!c->broke && n >= 2) {
    if (fabs(__dsub_rn(A[n - 1], 1.0)) < 1e-5) {
      if (np < c->mp) S[np] = (unsigned)c->plast;
      ++np;
    } else {
      bad = true;
    }
  }
  if (np != c->mp) bad = true;
  c->npush = np;
  if (bad) atomicOr(err, FRICC_DEV_PIVOTAL);
}

// the error word into a handle's status block, with |D| = m ("largest")
__global__ void k_put_meta(int64_t nd, const unsigned* err, unsigned long long* meta) {
  meta[0] = (unsigned long long)nd;
  meta[1] |= (unsigned long long)*err;
}

inline unsigned grid_for(int64_t n, int nt) {
  int64_t g = fricc_cdiv(n, nt);
  if (g > 152 * 32) g = 152 * 32;
  return (unsigned)(g < 1 ? 1 : g);
}

}  // namespace

// Scratch for one compression; everything comes from the stream-ordered pool.
struct CompressScratch {
  unsigned* hist = nullptr;
  unsigned* err = nullptr;
  unsigned long long* ckey = nullptr;
  unsigned* cidx = nullptr;
  unsigned long long* ktmp = nullptr;
  unsigned* vtmp = nullptr;
  unsigned* rhist = nullptr;
  unsigned long long* tstate = nullptr;
  unsigned* ticket = nullptr;
  double* dzero = nullptr;
  double* psum = nullptr;
  unsigned* bar = nullptr;
  double* Rb = nullptr;
  unsigned long long* ffail = nullptr;
  unsigned* S = nullptr;
  unsigned* S2 = nullptr;
  double* P = nullptr;
  Ctl* ctl = nullptr;
  Ctl* ctl2 = nullptr;  // a paired compression's second state
  exact::ChainScratch chain;
};

static void free_scratch(CompressScratch& s, cudaStream_t st) {
  fricc_free(s.hist, st);
  fricc_free(s.err, st);
  fricc_free(s.ckey, st);
  fricc_free(s.cidx, st);
  fricc_free(s.ktmp, st);
  fricc_free(s.vtmp, st);
  fricc_free(s.rhist, st);
  fricc_free(s.tstate, st);
  fricc_free(s.ticket, st);
  fricc_free(s.dzero, st);
  fricc_free(s.psum, st);
  fricc_free(s.bar, st);
  fricc_free(s.S2, st);
  fricc_free(s.ctl, st);
  fricc_free(s.ctl2, st);
  fricc_free(s.Rb, st);
  fricc_free(s.ffail, st);
  fricc_free(s.S, st);
  fricc_free(s.P, st);
  exact::free_chain(s.chain, st);
}

static int dev_status(unsigned e) {
  if (e & FRICC_DEV_P_GT_ONE) {
    fricc_set_error("ERROR MAKING PROBABILITY VECTOR: a sampling probability exceeds 1");
    return FRICC_ERR_P_GT_ONE;
  }
  if (e & FRICC_DEV_PIVOTAL) {
    fricc_set_error("ERROR IN PIVOTAL SAMPLING: acceptance probability outside [0, 1], leftover weight "
                    "|a - 1| >= 1e-5, or a wrong number of sampled elements");
    return FRICC_ERR_PIVOTAL;
  }
  if (e & FRICC_DEV_TIMEOUT) {
    fricc_set_error("a bounded device-side wait timed out");
    return FRICC_ERR_TIMEOUT;
  }
  if (e & FRICC_DEV_INDEX) {
    fricc_set_error("Indices are out of range for given tensor");
    return FRICC_ERR_INDEX;
  }
  return FRICC_OK;
}

// Compress x (device, n doubles) keeping m entries.  mode 0: "fri"
// (systematic, one uniform draw rn), mode 1: "largest".  Writes flat[m],
// vals[m] (device).  Every decision between phases (select digit, candidate
// count, |D|, R, the D threshold) stays on the device, so the only host
// round trip is the final one: with n_largest != nullptr the call
// synchronises the stream, reads |D| and the error word and reports them;
// with n_largest == nullptr it returns at once (nothing read back).
int fricc_glibc_uniforms_device(unsigned* hist, int64_t k, double* out, cudaStream_t st);

// ---------------------------------------------------------------------------
// parallel_sample (src/fri_utils.cpp:176-362): T chunks sampled pivotally,
// each walked by its own warp.  Per chunk (one block of 32): the reference's
// adjustment of the chunk's probabilities towards its integer count g (a
// running FP64 sum with a break; the per-element y is formed by every lane
// in parallel, only the running sum is sequential), then the pivotal weight
// walk of k_piv_chain on the adjusted probabilities.
struct SegInfo {
  int64_t lo, len;   // chunk position and length in q
  double t, a, qn;   // frac(a), a, the chunk's norm
  int64_t g;         // samples the chunk must give
};

__global__ void __launch_bounds__(32) k_seg_chain(const SegInfo* __restrict__ seg, double* __restrict__ P,
                                                  double* __restrict__ A, unsigned char* __restrict__ code,
                                                  Ctl* __restrict__ ctl) {
  const SegInfo sg = seg[blockIdx.x];
  Ctl* c = ctl + blockIdx.x;
  double* p = P + sg.lo;
  const int lane = threadIdx.x;
  const double gd = (double)sg.g;
  // 1. the adjustment (fri_utils.cpp:297-328): p_i <- y_i until the running sum
  //    crosses g, the crossing element taking the remainder
  const int mode = gd > sg.a ? 1 : (gd < sg.a ? -1 : 0);
  if (mode != 0) {
    double sj = sg.qn;
    bool done = false;
    for (int64_t i0 = 0; i0 < sg.len && !done; i0 += 32) {
      const int64_t i = i0 + lane;
      const double q = i < sg.len ? p[i] : 0.0;
      double y;
      if (mode > 0) {
        const double r = __ddiv_rn(q, sg.t);
        y = r < 1.0 ? r : 1.0;            // std::min(1., r): 1 unless r < 1 (NaN -> 1)
      } else {
        const double r = __ddiv_rn(__dsub_rn(q, sg.t), __dsub_rn(1.0, sg.t));
        y = 0.0 < r ? r : 0.0;            // std::max(0., r): r if 0 < r (NaN -> 0)
      }
      const double d = __dsub_rn(y, q);
      double myv = y;
      int hit = 32;
#pragma unroll
      for (int t = 0; t < 32; ++t) {
        const double dt = __shfl_sync(0xffffffffu, d, t);
        const double yt = __shfl_sync(0xffffffffu, y, t);
        if (i0 + t < sg.len && hit == 32) {
          sj = __dadd_rn(sj, dt);
          if (mode > 0 ? sj >= gd : sj <= gd) {
            hit = t;
            if (lane == t) myv = __dsub_rn(__dadd_rn(yt, gd), sj);
          }
        }
      }
      if (i < sg.len && lane <= hit) p[i] = myv;
      if (hit < 32) done = true;
    }
  }
  __syncwarp();
  // 2. the pivotal weight walk over the adjusted chunk (as k_piv_chain)
  const int64_t n = sg.len, mp = c->mp;
  double a = n > 0 ? p[0] : 0.0;
  if (lane == 0 && n > 0) {
    A[sg.lo] = a;
    code[sg.lo] = 0;
  }
  int64_t cnt = 0, jend = n - 1;
  int broke = 0;
  double pn = 1 + lane < n ? p[1 + lane] : 0.0;
  for (int64_t j0 = 1; j0 < n; j0 += 32) {
    const double pj = pn;
    const int64_t jn = j0 + 32 + lane;
    pn = jn < n ? p[jn] : 0.0;
    double myA = 0.0;
    bool myW = false;
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const double pt = __shfl_sync(0xffffffffu, pj, t);
      const double sum = __dadd_rn(a, pt);
      const bool w = !(sum < 1.0);
      a = w ? __dsub_rn(sum, 1.0) : sum;
      if (lane == t) {
        myA = a;
        myW = w;
      }
    }
    const int64_t j = j0 + lane;
    const bool valid = j < n;
    const unsigned wm = __ballot_sync(0xffffffffu, myW && valid);
    int stop = -1;
    if (mp == 0) {
      if (j0 == 1 && !(wm & 1u)) stop = 0;
    } else if (cnt < mp && cnt + __popc(wm) >= mp) {
      int64_t r = mp - cnt;
      for (int b = 0; b < 32; ++b)
        if (((wm >> b) & 1u) && --r == 0) {
          stop = b;
          break;
        }
    }
    if (valid && (stop < 0 || lane <= stop)) {
      A[sg.lo + j] = myA;
      code[sg.lo + j] = myW ? PV_EMIT : 0;
    }
    if (stop >= 0) {
      jend = j0 + stop;
      broke = 1;
      cnt = mp;
      break;
    }
    cnt += __popc(wm);
  }
  if (lane == 0) {
    c->jend = jend < 0 ? 0 : jend;
    c->npush = cnt;
    c->broke = broke;
  }
}

__global__ void k_s_to_flat(const unsigned* __restrict__ S, int64_t n, int64_t off, int64_t* __restrict__ out) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    out[k] = (int64_t)S[k] + off;
}

// the reference's sample_pivotal on the host, for the T chunk fractions
template <class Draw>
static int host_pivotal(int64_t n_sample, const std::vector<double>& probs, Draw draw, std::vector<int64_t>& S,
                        int64_t* used) {
  S.clear();
  *used = 0;
  const int64_t n = (int64_t)probs.size();
  if (n == 0) return n_sample == 0 ? FRICC_OK : FRICC_ERR_PIVOTAL;
  int64_t i = 0;
  double a = probs[0];
  for (int64_t j = 1; j < n; ++j) {
    a += probs[(size_t)j];
    const double r = draw();
    ++*used;
    if (a < 1.) {
      if (r < probs[(size_t)j] / a) i = j;
    } else {
      a -= 1.;
      const double pa = (1. - probs[(size_t)j]) / (1. - a);
      if (pa > 1 || pa < 0) return FRICC_ERR_PIVOTAL;
      if (r < pa) {
        S.push_back(i);
        i = j;
      } else {
        S.push_back(j);
      }
    }
    if ((int64_t)S.size() == n_sample) break;
    if (j == n - 1) {
      if (std::fabs(a - 1.) < 1e-5) S.push_back(i);
      else return FRICC_ERR_PIVOTAL;
    }
  }
  return (int64_t)S.size() == n_sample ? FRICC_OK : FRICC_ERR_PIVOTAL;
}

// glibc's rand() recurrence on a 31-word history (oldest first), on the host
static double host_glibc_uniform(unsigned* h) {
  const unsigned w = h[0] + h[28];
  for (int t = 0; t < 30; ++t) h[t] = h[t + 1];
  h[30] = w;
  return (double)(int)(w >> 1) / 2147483647.0;
}

// Steps of pivotal sampling after D, R and m' are on the device (ctl): the
// weight walk, the draws, the decisions, the scans; leaves S (m' indices).
// Phase timing of a compression (the reference's verbose table,
// src/fri_utils.cpp:509-519): CUDA events at the phase boundaries of the
// calling thread's compressions while enabled.  Boundaries: 0 start, 1 the
// largest elements and the remaining norm (the reference's "Sorting":
// get_d_largest), 2 the probability vector, 3 the samples, 4 the outputs
// ("Wrap up").
struct PhaseTimer {
  bool on = false;
  bool recorded = false;
  cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
};
static thread_local PhaseTimer g_phase;

static void phase_mark(int k, cudaStream_t st) {
  if (!g_phase.on) return;
  if (!g_phase.ev[k] && cudaEventCreate(&g_phase.ev[k]) != cudaSuccess) {
    g_phase.ev[k] = nullptr;
    return;
  }
  cudaEventRecord(g_phase.ev[k], st);
  if (k == 4) g_phase.recorded = true;
}

extern "C" int fricc_phase_timing_set(int on) {
  g_phase.on = on != 0;
  g_phase.recorded = false;
  return FRICC_OK;
}

// Seconds of each phase of the calling thread's last timed compression:
// sorting, P vector, sampling, wrap up, total (waits for its events).
extern "C" int fricc_phase_timing_read(double sec[5]) {
  if (!sec) {
    fricc_set_error("phase_timing_read: null output");
    return FRICC_ERR_ARG;
  }
  if (!g_phase.recorded) {
    fricc_set_error("phase_timing_read: no compression was timed on this thread");
    return FRICC_ERR_ARG;
  }
  float ms[5] = {0, 0, 0, 0, 0};
  FRICC_CUDA(cudaEventSynchronize(g_phase.ev[4]));
  for (int k = 0; k < 4; ++k) FRICC_CUDA(cudaEventElapsedTime(&ms[k], g_phase.ev[k], g_phase.ev[k + 1]));
  FRICC_CUDA(cudaEventElapsedTime(&ms[4], g_phase.ev[0], g_phase.ev[4]));
  for (int k = 0; k < 5; ++k) sec[k] = ms[k] * 1e-3;
  return FRICC_OK;
}

static int pivotal(int64_t n, const GenP& gp, Ctl* ctl, CompressScratch& s, unsigned* glibc_hist, int64_t* n_draws,
                   cudaStream_t st) {
  double *P = nullptr, *A = nullptr, *R = nullptr;
  unsigned char* code = nullptr;
  void* seg = nullptr;
  int64_t *tlast = nullptr, *tcnt = nullptr;
  const int64_t ntile = fricc_cdiv(n, PV_TILE);
  int rc = fricc_alloc_t(&P, n, st);
  if (!rc) rc = fricc_alloc_t(&A, n, st);
  if (!rc) rc = fricc_alloc_t(&code, n, st);
  if (!rc) rc = fricc_alloc_t(&tlast, ntile, st);
  if (!rc) rc = fricc_alloc_t(&tcnt, ntile, st);
  int64_t jend = 0;
  unsigned e = 0;
  if (!rc) {
    k_pvec<<<(unsigned)fricc_cdiv(n, exact::CH / PV_SUB), 256, 0, st>>>(gp, n, P, s.err, nullptr);
    phase_mark(2, st);
    PivSegs g;
    g.n = n;
    g.S = fricc_cdiv(n, PW_SEGS) > PW_MIN ? fricc_cdiv(fricc_cdiv(n, PW_SEGS), 32) * 32 : PW_MIN;
    g.nseg = fricc_cdiv(n, g.S);
    // one block for all of the segments' arrays: 8-byte items first
    const int64_t q = g.nseg;
    rc = fricc_alloc(&seg, (size_t)(q * (8 + 8 + 16 + 8 + 8) + (q + 2) * 4), st);
    if (!rc) {
      char* b = static_cast<char*>(seg);
      g.map = reinterpret_cast<exact::Map*>(b);
      g.f = reinterpret_cast<unsigned long long*>(b + 16 * q);
      g.start = reinterpret_cast<int64_t*>(b + 24 * q);
      g.claim = reinterpret_cast<double*>(b + 32 * q);
      g.end = reinterpret_cast<double*>(b + 40 * q);
      g.cnt = reinterpret_cast<int*>(b + 48 * q);
      const unsigned gw = (unsigned)fricc_cdiv(g.nseg, 64);
      k_piv_sums<<<grid_for(g.nseg, 8), 256, 0, st>>>(P, g, ctl);
      k_piv_prefix<<<1, 1024, 0, st>>>(g, ctl);
      k_piv_starts<<<gw, 64, 0, st>>>(P, g, ctl);
      k_piv_walk<1><<<gw, 64, 0, st>>>(P, g, ctl, A, code, 0);
      for (int round = 0; round < 3; ++round) {
        k_piv_claims<<<1, 1024, 0, st>>>(g, ctl, round);
        k_piv_walk<2><<<gw, 64, 0, st>>>(P, g, ctl, A, code, round);
      }
      k_piv_end<<<1, 1024, 0, st>>>(g, code, ctl);
      k_piv_chain<<<1, 32, 0, st>>>(P, n, ctl, A, code);
      fricc_note_launch(13);
    }
  }
  if (!rc) {
    rc = fricc_cuda_check(cudaGetLastError(), "pivotal chain");
  }
  if (!rc) rc = fricc_cuda_check(cudaMemcpyAsync(&jend, &ctl->jend, sizeof(int64_t), cudaMemcpyDeviceToHost, st), "jend");
  if (!rc) rc = fricc_cuda_check(cudaMemcpyAsync(&e, s.err, sizeof(unsigned), cudaMemcpyDeviceToHost, st), "err");
  if (!rc) rc = fricc_cuda_check(cudaStreamSynchronize(st), "pivotal chain");
  if (!rc) rc = dev_status(e);  // p > 1: the reference exits before drawing
  const int64_t used = jend;   // one draw per visited element j = 1..jend
  if (!rc && used > 0) {
    rc = fricc_alloc_t(&R, used, st);
    if (!rc && glibc_hist) {
      rc = fricc_glibc_uniforms_device(glibc_hist, used, R, st);
    } else if (!rc) {
      std::vector<double> h((size_t)used);
      for (int64_t k = 0; k < used; ++k) h[(size_t)k] = (double)rand() / RAND_MAX;
      rc = fricc_cuda_check(cudaMemcpyAsync(R, h.data(), sizeof(double) * (size_t)used, cudaMemcpyHostToDevice, st),
                            "draws");
      if (!rc) rc = fricc_cuda_check(cudaStreamSynchronize(st), "draws");
    }
  }
  if (!rc) {
    if (n_draws) *n_draws = used;
    if (used > 0) k_piv_decide<<<grid_for(used, 256), 256, 0, st>>>(P, A, code, R, ctl, s.err);
    k_piv_tiles<<<(unsigned)ntile, PV_NT, 0, st>>>(code, ctl, tlast, tcnt);
    k_piv_carry<<<1, 1024, 0, st>>>(tlast, tcnt, ntile, ctl);
    k_piv_emit<<<(unsigned)ntile, PV_NT, 0, st>>>(code, tlast, tcnt, ctl, s.S);
    k_piv_final<<<1, 1, 0, st>>>(A, n, ctl, s.S, s.err);
    fricc_note_launch(used > 0 ? 5 : 4);
    rc = fricc_cuda_check(cudaGetLastError(), "pivotal");
  }
  if (!rc) rc = fricc_cuda_check(cudaMemcpyAsync(&e, s.err, sizeof(unsigned), cudaMemcpyDeviceToHost, st), "err");
  if (!rc) rc = fricc_cuda_check(cudaStreamSynchronize(st), "pivotal");
  if (!rc) rc = dev_status(e);
  fricc_free(P, st);
  fricc_free(A, st);
  fricc_free(R, st);
  fricc_free(code, st);
  fricc_free(seg, st);
  fricc_free(tlast, st);
  fricc_free(tcnt, st);
  return rc;
}

// The uniform draws of a compression and (paired) of its second one: host
// values, or device words (replica r's at a_dev[r * stride]).
struct Draws {
  double a = 0.0, b = 0.0;
  const double* a_dev = nullptr;
  const double* b_dev = nullptr;
  int64_t stride = 0;
};

// One compression's (or a batch of R's) first half: scratch, histogram,
// one_norm, candidates, their sort, and for mode 0 and 2 the
// remaining-norm chain: |D|, R and m' in s.ctl (and s.ctl2 when paired).
static int compress_front(const double* x, int64_t n, int64_t m, int R, int mode, bool paired, const Draws& dr,
                          const Rep& rp, CompressScratch& s, cudaStream_t st) {
  const int64_t ntile = fricc_cdiv(n, 4096);
  const int64_t nch_n = fricc_cdiv(n, exact::CH), nch_m = fricc_cdiv(m, exact::CH);
  const int64_t nch1 = (nch_n > nch_m ? nch_n : nch_m) + 1;
  const int64_t rhw = radix::hist_words(n);
  const size_t r_ = (size_t)R;
  const bool fri = mode != 1;
  int rc = fricc_alloc_t(&s.ctl, r_, st);
  if (!rc && paired) rc = fricc_alloc_t(&s.ctl2, r_, st);
  if (!rc) rc = fricc_alloc_t(&s.hist, r_ * NDIG, st);
  if (!rc) rc = fricc_alloc_t(&s.err, r_, st);
  if (!rc) rc = fricc_alloc_t(&s.ckey, r_ * n, st);
  if (!rc) rc = fricc_alloc_t(&s.cidx, r_ * n, st);
  if (!rc) rc = fricc_alloc_t(&s.ktmp, r_ * n, st);
  if (!rc) rc = fricc_alloc_t(&s.vtmp, r_ * n, st);
  if (!rc) rc = fricc_alloc_t(&s.tstate, r_ * (ntile + 1), st);  // + a zero word no tile writes (the test-only wait)
  if (!rc) rc = fricc_alloc_t(&s.ticket, r_, st);
  if (!rc) rc = fricc_alloc_t(&s.rhist, r_ * rhw, st);
  if (!rc) rc = fricc_alloc_t(&s.bar, 1, st);
  if (!rc) rc = fricc_alloc_t(&s.dzero, 1, st);
  if (!rc) rc = fricc_alloc_t(&s.ffail, r_, st);
  if (!rc) rc = fricc_alloc_t(&s.psum, r_ * nch1, st);
  if (!rc && fri) rc = exact::chain_scratch(s.chain, R * nch1, st, R);
  if (!rc && fri) rc = fricc_alloc_t(&s.Rb, r_ * (m + 1), st);
  if (!rc && fri) rc = fricc_alloc_t(&s.S, r_ * m, st);
  if (!rc && paired) rc = fricc_alloc_t(&s.S2, r_ * m, st);
  if (rc) return rc;

  k_init<<<dim3(grid_for(fri ? m : NDIG, 512), R), 256, 0, st>>>(s.hist, s.tstate, ntile + 1, s.S, s.S2, m, s.ctl,
                                                                 dr.a, dr.a_dev, dr.stride, s.err, s.ticket, s.ffail,
                                                                 s.dzero, s.bar, s.psum, nch_n + 1);
  phase_mark(0, st);
  const int bits = select_bits();
  const int64_t gh = nch_n < 152 * 6 ? nch_n : 152 * 6;
  k_hist_sums<<<dim3((unsigned)gh, R), 256, sizeof(unsigned) << bits, st>>>(x, n, s.hist, bits,
                                                                            fri ? s.chain.csum : nullptr, rp);
  fricc_note_launch(2);
  const int64_t cw = (int64_t)(sizeof(Ctl) / sizeof(int64_t));  // a Ctl in 8-byte words
  static_assert(sizeof(Ctl) % sizeof(int64_t) == 0, "Ctl must be a whole number of int64 words");
  exact::ChainStride zero_start, ctl_start;
  ctl_start.s_init = cw;
  if (fri) {  // one_norm
    rc = exact::run_chain<GenAbs, exact::ConsNull, false>(GenAbs{x, rp.n}, exact::Len{n}, s.dzero, false,
                                                          exact::ConsNull{}, s.chain, st, R, zero_start, true,
                                                          &s.ctl->norm, cw);
    if (rc) return rc;
  }
  k_select_digit<<<R, 1024, 0, st>>>(s.hist, m, s.ctl, bits, fri ? 1 : 0, rp);
  k_compact<<<dim3((unsigned)ntile, R), 256, 0, st>>>(x, n, s.ctl, s.ktmp, s.vtmp, s.tstate, s.ticket, s.err,
                                                      s.tstate + ntile,
                                                      (long long)fricc_tune_get(FRICC_TUNE_TEST_WAIT), 63 - bits, rp);
  fricc_note_launch(2);
  // argsort (src/fri_utils.cpp:11-36) of the candidates
  radix::Batch bt;
  bt.kv_stride = rp.n;
  bt.hist_stride = rhw;
  bt.n_stride = cw;
  rc = radix::sort_desc_dev(s.ktmp, s.vtmp, s.ckey, s.cidx, n, &s.ctl->ncand, s.rhist, s.bar, s.err, st, R, bt);
  if (rc || !fri) return rc;

  const ConsAccept ca{m, s.Rb, s.ffail, s.ctl, rp.one};
  k_rem_first<<<R, 1024, 0, st>>>(ca, s.ckey, s.cidx, s.ctl, rp);
  fricc_note_launch();
  exact::Len ln;
  ln.n = m;
  ln.dev = &s.ctl->mchain;
  ln.stride = cw;
  ln.skip = reinterpret_cast<const int*>(&s.ctl->found);
  ln.sstride = 2 * cw;
  if (m > REM_CHUNKS * exact::CH) {
    rc = exact::run_chain<GenSorted, ConsAccept, true>(GenSorted{s.ckey, rp.n}, ln, &s.ctl->norm, true, ca, s.chain,
                                                       st, R, ctl_start);
    if (rc) return rc;
  }
  if (m > REM_CHUNKS * exact::CH || paired) {
    k_finish_d<<<R, 1, 0, st>>>(s.ffail, s.Rb, s.ckey, s.cidx, m, s.ctl, s.ctl2, dr.b, dr.b_dev, dr.stride, rp);
    fricc_note_launch();
  }
  return fricc_cuda_check(cudaGetLastError(), "compression");
}

// Probabilities (once, with the p > 1 check), their exact partial sums and
// the systematic samples of one or (s.ctl2) both draws.  With m' = 0 every p
// is 0 (or NaN); with R <= 0 or not finite no interval matches: in both
// cases all samples keep index 0, as in the reference.
static int compress_systematic(const double* x, int64_t n, int64_t m, int R, const Rep& rp, CompressScratch& s,
                               cudaStream_t st) {
  int rc = fricc_alloc_t(&s.P, (size_t)R * n, st);
  if (rc) return rc;
  k_pvec<<<dim3((unsigned)fricc_cdiv(n, exact::CH / PV_SUB), R), 256, 0, st>>>(GenP{x, s.ctl, rp.n, rp.one}, n, s.P,
                                                                               s.err, s.psum, rp);
  fricc_note_launch();
  phase_mark(2, st);
  const GenPv gpv{s.P, x, s.ctl, rp.n, rp.one};
  const ConsSample cs{s.ctl, s.S, rp.one, rp.m};
  exact::ChainScratch sc = s.chain;  // the same scratch, with the chunk sums k_pvec left
  sc.csum = s.psum;
  if (s.ctl2)
    return exact::run_chain<GenPv, ConsSample2, true>(gpv, exact::Len{n}, s.dzero, false,
                                                      ConsSample2{cs, ConsSample{s.ctl2, s.S2, rp.one, rp.m}}, sc, st,
                                                      R, exact::ChainStride{}, true);
  return exact::run_chain<GenPv, ConsSample, true>(gpv, exact::Len{n}, s.dzero, false, cs, sc, st, R,
                                                   exact::ChainStride{}, true);
}

// mode 2: "fri" with pivotal sampling.  Its draws (one per visited element)
// come from the glibc stream whose history is glibc_hist[31] (host, oldest
// first; advanced past the draws on return), or with glibc_hist == nullptr
// from this process's own rand(), as the reference draws them.  *n_draws
// receives the number consumed.  Synchronises the stream twice (the number
// of draws, then the result).
// meta (device, 2 words, optional): receives |D| and ORs in the error bits,
// in stream order, so a caller that passes n_largest == nullptr never waits.
int fricc_compress_device(const double* x, int64_t n, int64_t m, int mode, double rn, cudaStream_t st,
                          int64_t* flat, double* vals, int64_t* n_largest, unsigned* glibc_hist, int64_t* n_draws,
                          unsigned long long* meta, const double* rn_dev, const CompressPairOut* pair) {
  if (pair && (mode != 0 || !meta || !pair->flat || !pair->vals || !pair->meta)) {
    fricc_set_error("compress: a paired compression is systematic FRI with status blocks");
    return FRICC_ERR_ARG;
  }
  if (n < 0 || m <= 0 || m > n) {
    fricc_set_error("Bad m_keep value: need 0 < m <= tensor size (m=%lld, size=%lld)", (long long)m,
                    (long long)n);
    return FRICC_ERR_ARG;
  }
  if (n >= 0xffffffffLL) {
    fricc_set_error("tensor too large for 32-bit indices (%lld elements)", (long long)n);
    return FRICC_ERR_ARG;
  }
  CompressScratch s;
  int rc = FRICC_OK;
#define TRY(x)                  \
  do {                          \
    rc = (x);                   \
    if (rc) goto done;          \
  } while (0)

  {
    Draws dr;
    dr.a = rn;
    dr.a_dev = rn_dev;
    if (pair) {
      dr.b = pair->rn;
      dr.b_dev = pair->rn_dev;
    }
    TRY(compress_front(x, n, m, 1, mode, pair != nullptr, dr, Rep{}, s, st));
    if (mode == 1) {  // "largest": argsort(x, m) with unscaled values
      phase_mark(1, st);
      phase_mark(2, st);
      phase_mark(3, st);
      k_out_d<<<grid_for(m, 256), 256, 0, st>>>(x, s.cidx, m, flat, vals);
      fricc_note_launch();
      phase_mark(4, st);
      if (meta) {
        k_put_meta<<<1, 1, 0, st>>>(m, s.err, meta);
        fricc_note_launch();
      }
      TRY(fricc_cuda_check(cudaGetLastError(), "largest"));
      if (n_largest) {
        unsigned e = 0;
        TRY(fricc_cuda_check(cudaMemcpyAsync(&e, s.err, sizeof(unsigned), cudaMemcpyDeviceToHost, st), "err"));
        TRY(fricc_cuda_check(cudaStreamSynchronize(st), "compression"));
        TRY(dev_status(e));
        *n_largest = m;
      }
      goto done;
    }
    phase_mark(1, st);
    const GenP gp{x, s.ctl};
    if (mode == 2) {
      TRY(pivotal(n, gp, s.ctl, s, glibc_hist, n_draws, st));
      phase_mark(3, st);
      k_out<GenP><<<grid_for(m, 256), 256, 0, st>>>(gp, n, s.cidx, s.S, m, flat, vals, s.err, meta);
      fricc_note_launch();
      phase_mark(4, st);
    } else {
      TRY(compress_systematic(x, n, m, 1, Rep{}, s, st));
      phase_mark(3, st);
      k_out<GenPv><<<grid_for(m, 256), 256, 0, st>>>(GenPv{s.P, x, s.ctl}, n, s.cidx, s.S, m, flat, vals, s.err,
                                                         meta);
      if (pair)
        k_out<GenPv><<<grid_for(m, 256), 256, 0, st>>>(GenPv{s.P, x, s.ctl2}, n, s.cidx, s.S2, m, pair->flat,
                                                           pair->vals, s.err, pair->meta);
      fricc_note_launch(pair ? 2 : 1);
      phase_mark(4, st);
    }
    TRY(fricc_cuda_check(cudaGetLastError(), "output"));
    if (n_largest) {
      unsigned e = 0;
      int64_t nd = 0;
      TRY(fricc_cuda_check(cudaMemcpyAsync(&e, s.err, sizeof(unsigned), cudaMemcpyDeviceToHost, st), "err"));
      TRY(fricc_cuda_check(cudaMemcpyAsync(&nd, &s.ctl->nd, sizeof(int64_t), cudaMemcpyDeviceToHost, st), "nd"));
      TRY(fricc_cuda_check(cudaStreamSynchronize(st), "compression"));
      TRY(dev_status(e));
      *n_largest = nd;
    }
  }
done:
#undef TRY
  free_scratch(s, st);
  return rc;
}

// ---------------------------------------------------------------------------
// Replica batches: the paired systematic compression of R tensors of one
// shape (replica r's tensor x + r n) in one set of launches -- every kernel
// of the single path with the replica on its grid's y (or x) dimension, each
// replica's arithmetic that of its own single compression, so each output is
// bit for bit the one fricc_sp_recompress_pair would give.
int fricc_compress_pair_batch_device(const double* x, int64_t n, int64_t m, int R, const double* rn_dev,
                                     int64_t* flatA, double* valsA, unsigned long long* metaA, int64_t* flatB,
                                     double* valsB, unsigned long long* metaB, cudaStream_t st) {
  if (!x || !rn_dev || !flatA || !valsA || !metaA || !flatB || !valsB || !metaB || R < 1 || R > 65535) {
    fricc_set_error("compress batch: bad arguments");
    return FRICC_ERR_ARG;
  }
  if (n <= 0 || m <= 0 || m > n || n >= 0xffffffffLL) {
    fricc_set_error("Bad m_keep value: need 0 < m <= tensor size < 2^32 (m=%lld, size=%lld)", (long long)m,
                    (long long)n);
    return FRICC_ERR_ARG;
  }
  Rep rp;
  rp.n = n;
  rp.m = m;
  rp.tile = fricc_cdiv(n, 4096) + 1;
  rp.one = 1;
  CompressScratch s;
  Draws dr;
  dr.a_dev = rn_dev;
  dr.b_dev = rn_dev + 1;
  dr.stride = 2;
  int rc = compress_front(x, n, m, R, 0, true, dr, rp, s, st);
  if (!rc) rc = compress_systematic(x, n, m, R, rp, s, st);
  if (!rc) {
    const dim3 g(grid_for(m, 256), R);
    k_out<GenPv><<<g, 256, 0, st>>>(GenPv{s.P, x, s.ctl, n, 1}, n, s.cidx, s.S, m, flatA, valsA, s.err, metaA, rp);
    k_out<GenPv><<<g, 256, 0, st>>>(GenPv{s.P, x, s.ctl2, n, 1}, n, s.cidx, s.S2, m, flatB, valsB, s.err, metaB, rp);
    fricc_note_launch(2);
    rc = fricc_cuda_check(cudaGetLastError(), "compress batch");
  }
  free_scratch(s, st);
  return rc;
}

// Unpack the flat indices of R compressions (m each, stacked) into slots;
// an out-of-range index is ORed into the replica's meta[1].
int fricc_unpack_batch_async(const int64_t* flat, int64_t m, int R, const int64_t dims[4], int* slots,
                             unsigned long long* meta, cudaStream_t st) {
  Rep rp;
  rp.m = m;
  rp.one = 1;
  k_unpack<<<dim3(grid_for(m, 256), R), 256, 0, st>>>(flat, m, dims[0], dims[1], dims[2], dims[3], slots,
                                                      reinterpret_cast<unsigned*>(meta + 1), rp);
  fricc_note_launch();
  return fricc_cuda_check(cudaGetLastError(), "unpack batch");
}

// The error bits of a deferred status word, as a status code (and message).
int fricc_dev_status(unsigned e) { return dev_status(e); }

// Unpack without waiting: an out-of-range index is ORed into meta[1].
int fricc_unpack_async(const int64_t* flat, int64_t m, const int64_t dims[4], int* slots, unsigned long long* meta,
                       cudaStream_t st) {
  k_unpack<<<grid_for(m, 256), 256, 0, st>>>(flat, m, dims[0], dims[1], dims[2], dims[3], slots,
                                             reinterpret_cast<unsigned*>(meta + 1));
  fricc_note_launch();
  return fricc_cuda_check(cudaGetLastError(), "unpack");
}

int fricc_unpack_device(const int64_t* flat, int64_t m, const int64_t dims[4], int* slots, cudaStream_t st) {
  unsigned* err = nullptr;
  int rc = fricc_alloc_t(&err, 1, st);
  if (rc) return rc;
  cudaMemsetAsync(err, 0, sizeof(unsigned), st);
  k_unpack<<<grid_for(m, 256), 256, 0, st>>>(flat, m, dims[0], dims[1], dims[2], dims[3], slots, err);
  fricc_note_launch();
  unsigned e = 0;
  cudaMemcpyAsync(&e, err, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  cudaError_t ce = cudaStreamSynchronize(st);
  fricc_free(err, st);
  if (ce != cudaSuccess) return fricc_cuda_fail(ce, "unpack", __FILE__, __LINE__);
  return dev_status(e);
}

namespace {
struct ConsWrite {
  double* out;
  __device__ __forceinline__ void operator()(int64_t i, double, double after, double) const { out[i] = after; }
};
}  // namespace

// out[i] = fl(out[i-1] + |x_i|), out[-1] = 0: the running sums of one_norm
// (src/fri_utils.cpp:164-171) / std::partial_sum (:142-143), bit for bit.
int fricc_seq_cumsum_device(const double* x, int64_t n, double* out, cudaStream_t st) {
  if (n < 0 || (n > 0 && (!x || !out))) {
    fricc_set_error("seq_cumsum: bad arguments");
    return FRICC_ERR_ARG;
  }
  if (n == 0) return FRICC_OK;
  exact::ChainScratch sc;
  double* dzero = nullptr;
  int rc = fricc_alloc_t(&dzero, 1, st);
  if (!rc) {
    cudaMemsetAsync(dzero, 0, sizeof(double), st);
    rc = exact::run_chain<GenAbs, ConsWrite, true>(GenAbs{x}, exact::Len{n}, dzero, false, ConsWrite{out}, sc, st);
  }
  exact::free_chain(sc, st);
  fricc_free(dzero, st);
  return rc;
}

// The chunk walks, the chunk draws (in chunk order), the decisions and the
// scans of each chunk, S assembled in the reference's order.
static int fricc_parallel_sample_finish(const double* q, int64_t n, int64_t n_sample, std::vector<SegInfo>& seg,
                                        unsigned* glibc_hist, int64_t* S_out, int64_t* n_draws, int64_t used,
                                        unsigned* err, cudaStream_t st) {
  const int T = (int)seg.size();
  double *P = nullptr, *A = nullptr, *R = nullptr;
  unsigned char* code = nullptr;
  unsigned* Sseg = nullptr;
  SegInfo* dseg = nullptr;
  Ctl* ctl = nullptr;
  int64_t *tlast = nullptr, *tcnt = nullptr;
  std::vector<Ctl> hc((size_t)T);
  std::vector<int64_t> dbase((size_t)T + 1, 0);
  unsigned e = 0;
  int64_t maxlen = 0;
  for (auto& g : seg) maxlen = g.len > maxlen ? g.len : maxlen;
  const int64_t ntile_max = fricc_cdiv(maxlen, PV_TILE);
  int rc = fricc_alloc_t(&P, n, st);
  if (!rc) rc = fricc_alloc_t(&A, n, st);
  if (!rc) rc = fricc_alloc_t(&code, n, st);
  if (!rc) rc = fricc_alloc_t(&Sseg, n_sample > 0 ? n_sample : 1, st);
  if (!rc) rc = fricc_alloc_t(&dseg, T, st);
  if (!rc) rc = fricc_alloc_t(&ctl, T, st);
  if (!rc) rc = fricc_alloc_t(&tlast, ntile_max, st);
  if (!rc) rc = fricc_alloc_t(&tcnt, ntile_max, st);
  if (!rc) {
    for (int j = 0; j < T; ++j) {
      std::memset(&hc[(size_t)j], 0, sizeof(Ctl));
      hc[(size_t)j].mp = seg[(size_t)j].g;
    }
    cudaError_t ce = cudaMemcpyAsync(P, q, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(dseg, seg.data(), sizeof(SegInfo) * T, cudaMemcpyHostToDevice, st);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(ctl, hc.data(), sizeof(Ctl) * T, cudaMemcpyHostToDevice, st);
    if (ce == cudaSuccess) {
      k_seg_chain<<<(unsigned)T, 32, 0, st>>>(dseg, P, A, code, ctl);
      fricc_note_launch();
      ce = cudaGetLastError();
    }
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(hc.data(), ctl, sizeof(Ctl) * T, cudaMemcpyDeviceToHost, st);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
    if (ce != cudaSuccess) rc = fricc_cuda_fail(ce, "parallel_sample walk", __FILE__, __LINE__);
  }
  if (!rc) {
    // chunk j consumes one draw per element it visits after its first
    for (int j = 0; j < T; ++j) dbase[(size_t)j + 1] = dbase[(size_t)j] + (seg[(size_t)j].len >= 2 ? hc[(size_t)j].jend : 0);
    const int64_t total = dbase[(size_t)T];
    if (total > 0) {
      rc = fricc_alloc_t(&R, total, st);
      if (!rc && glibc_hist) {
        rc = fricc_glibc_uniforms_device(glibc_hist, total, R, st);
      } else if (!rc) {
        std::vector<double> h((size_t)total);
        for (auto& r : h) r = (double)rand() / RAND_MAX;
        rc = fricc_cuda_check(cudaMemcpyAsync(R, h.data(), sizeof(double) * total, cudaMemcpyHostToDevice, st),
                              "draws");
        if (!rc) rc = fricc_cuda_check(cudaStreamSynchronize(st), "draws");
      }
    }
    used += total;
  }
  if (!rc) {
    int64_t lb = 0;
    for (int j = 0; j < T && !rc; ++j) {
      const SegInfo& g = seg[(size_t)j];
      Ctl* cj = ctl + j;
      const int64_t nt = fricc_cdiv(g.len, PV_TILE);
      if (hc[(size_t)j].jend > 0)
        k_piv_decide<<<grid_for(hc[(size_t)j].jend, 256), 256, 0, st>>>(P + g.lo, A + g.lo, code + g.lo,
                                                                        R + dbase[(size_t)j], cj, err);
      k_piv_tiles<<<(unsigned)nt, PV_NT, 0, st>>>(code + g.lo, cj, tlast, tcnt);
      k_piv_carry<<<1, 1024, 0, st>>>(tlast, tcnt, nt, cj);
      k_piv_emit<<<(unsigned)nt, PV_NT, 0, st>>>(code + g.lo, tlast, tcnt, cj, Sseg + lb);
      k_piv_final<<<1, 1, 0, st>>>(A + g.lo, g.len, cj, Sseg + lb, err);
      if (g.g > 0) k_s_to_flat<<<grid_for(g.g, 256), 256, 0, st>>>(Sseg + lb, g.g, g.lo, S_out + lb);
      fricc_note_launch(6);
      lb += g.g;
      rc = fricc_cuda_check(cudaGetLastError(), "parallel_sample");
    }
  }
  if (!rc) rc = fricc_cuda_check(cudaMemcpyAsync(&e, err, sizeof(unsigned), cudaMemcpyDeviceToHost, st), "err");
  if (!rc) rc = fricc_cuda_check(cudaStreamSynchronize(st), "parallel_sample");
  if (!rc) rc = dev_status(e);
  if (!rc && n_draws) *n_draws = used;
  fricc_free(P, st);
  fricc_free(A, st);
  fricc_free(R, st);
  fricc_free(code, st);
  fricc_free(Sseg, st);
  fricc_free(dseg, st);
  fricc_free(ctl, st);
  fricc_free(tlast, st);
  fricc_free(tcnt, st);
  fricc_free(err, st);
  return rc;
}

// parallel_sample with T chunks over q (device, n doubles): S (device, n_sample
// int64) in the reference's order; draws from glibc_hist (host, advanced) or
// from this process's rand(), taken in chunk order.  *n_draws: draws used.
int fricc_parallel_sample_device(const double* q, int64_t n, int64_t n_sample, int T, unsigned* glibc_hist,
                                 int64_t* S_out, int64_t* n_draws, cudaStream_t st) {
  if (!q || !S_out || n <= 0 || n_sample < 0 || T < 1 || n < T || n >= 0xffffffffLL) {
    fricc_set_error("parallel_sample: bad arguments (need 1 <= chunks <= n, n < 2^32)");
    return FRICC_ERR_ARG;
  }
  const int64_t step = n / T;
  std::vector<SegInfo> seg((size_t)T);
  std::vector<double> frac((size_t)T);
  int rc = FRICC_OK;
  double *d_norm = nullptr, *dzero = nullptr;
  unsigned* err = nullptr;
  exact::ChainScratch sc;
  int64_t used = 0;
#define PTRY(x)           \
  do {                    \
    rc = (x);             \
    if (rc) goto pdone;   \
  } while (0)
  {
    // norms: exact sequential sums (the reference's one_norm at one thread)
    PTRY(fricc_alloc_t(&d_norm, T + 1, st));
    PTRY(fricc_alloc_t(&dzero, 1, st));
    PTRY(fricc_alloc_t(&err, 1, st));
    PTRY(fricc_cuda_check(cudaMemsetAsync(dzero, 0, sizeof(double), st), "memset"));
    PTRY(fricc_cuda_check(cudaMemsetAsync(err, 0, sizeof(unsigned), st), "memset"));
    for (int j = 0; j <= T; ++j) {
      const int64_t lo = j < T ? j * step : 0, hi = j < T ? ((j + 1 == T) ? n : lo + step) : n;
      PTRY((exact::run_chain<GenAbs, exact::ConsNull, false>(GenAbs{q + lo}, exact::Len{hi - lo}, dzero, false,
                                                              exact::ConsNull{}, sc, st, 1, exact::ChainStride{},
                                                              false, d_norm + j)));
    }
    std::vector<double> hn((size_t)T + 1);
    PTRY(fricc_cuda_check(cudaMemcpyAsync(hn.data(), d_norm, sizeof(double) * (T + 1), cudaMemcpyDeviceToHost, st),
                          "norms"));
    PTRY(fricc_cuda_check(cudaStreamSynchronize(st), "norms"));
    const double q_norm = hn[(size_t)T];
    uint64_t c = (uint64_t)n_sample;
    for (int j = 0; j < T; ++j) {
      SegInfo& g = seg[(size_t)j];
      g.lo = j * step;
      g.len = (j + 1 == T) ? n - g.lo : step;
      g.qn = hn[(size_t)j];
      g.a = (double)(uint64_t)n_sample * g.qn / q_norm;
      g.t = g.a - std::floor(g.a);
      g.g = (int)std::floor(g.a);
      frac[(size_t)j] = g.t;
      c -= (uint64_t)(int64_t)(int)g.g;
    }
    if (c > (uint64_t)T) {
      fricc_set_error("ERROR IN PIVOTAL SAMPLING: chunk counts exceed n_sample");
      PTRY(FRICC_ERR_PIVOTAL);
    }
    // the fraction sample decides which chunks give one more; its draws come
    // first, one at a time, from the same stream
    std::vector<int64_t> sp;
    int64_t uf = 0;
    auto draw = [&]() { return glibc_hist ? host_glibc_uniform(glibc_hist) : (double)rand() / RAND_MAX; };
    rc = host_pivotal((int64_t)c, frac, draw, sp, &uf);
    if (rc) {
      fricc_set_error("ERROR IN PIVOTAL SAMPLING (chunk fractions)");
      goto pdone;
    }
    used += uf;
    for (int64_t k : sp) seg[(size_t)k].g += 1;
    for (auto& g : seg)
      if (g.g < 0 || g.g > g.len) {
        fricc_set_error("ERROR IN PIVOTAL SAMPLING: a chunk cannot give its %lld samples", (long long)g.g);
        PTRY(FRICC_ERR_PIVOTAL);
      }
  }
pdone:
#undef PTRY
  exact::free_chain(sc, st);
  fricc_free(d_norm, st);
  fricc_free(dzero, st);
  if (rc) {
    fricc_free(err, st);
    return rc;
  }
  return fricc_parallel_sample_finish(q, n, n_sample, seg, glibc_hist, S_out, n_draws, used, err, st);
}
