// Exact, parallel reproduction of a SEQUENTIAL left-to-right FP64 sum of
// non-negative addends (or of a chain of subtractions of them), i.e. the
// bits of
//     s_0 = s_init;  s_{i+1} = fl(s_i + a_i)   (or fl(s_i - a_i))
// for i = 0..len-1, as a single CPU thread computes them.
//
// FRI compression needs three such chains bit for bit (fri-cc
// src/fri_utils.cpp): one_norm (:164-171), the remaining-norm chain
// R -= |x_(d)| of get_d_largest (:411-421), and std::partial_sum(p) of
// sample_systematic (:142-143).  A parallel reduction rounds differently,
// so instead:
//
// * Inside one binade [2^e, 2^(e+1)) every double is n * ulp with an
//   integer n in [2^52, 2^53] (the bottom binade, which includes the
//   subnormals, is [0, 2^-1021) with n in [0, 2^53]).  Adding a >= 0 moves
//   n by q = floor(a/ulp) plus a rounding carry that depends only on the
//   remainder class of a (0, <1/2, =1/2, >1/2) and, for exact ties, on the
//   parity of n.  A step is therefore a map n -> n + (n odd ? d1 : d0),
//   and such maps compose associatively: the chain inside a binade is a
//   parallel scan over pairs of int64.
// * The binade of the running sum is predicted from an approximate
//   (parallel) prefix sum with a safety margin; chunks whose predicted
//   range stays inside one binade are "clean".
// * A chunk whose predicted range crosses binades (the first one crosses a
//   dozen) is cut at the elements whose step may leave a binade: the maps of the
//   segments between them come from one segmented scan, and the cuts are
//   single steps of real FP64 additions.
// * A single-block walk applies the chunk maps to the exact running value,
//   verifies every assumption (start in the predicted binade, end inside
//   it) and, where one fails, processes that chunk exactly: scan under the current binade, find the first
//   element whose step would leave it, perform that one step with a real
//   FP64 add, continue.  Correctness never depends on the prediction.
#pragma once
#include <climits>
#include <type_traits>
#include <utility>

#include "common.cuh"

namespace exact {

// Replica batches: a chain can run for R independent sequences at once
// (blockIdx.y, or blockIdx.x for the one-block kernels, is the replica).  A
// generator or consumer with a method at(r) gives replica r's copy (its
// pointers moved to that replica's data); one without is shared by all.
template <class G, class = void>
struct has_at : std::false_type {};
template <class G>
struct has_at<G, std::void_t<decltype(std::declval<const G&>().at(0))>> : std::true_type {};
template <class G>
__device__ __forceinline__ G replica_of(const G& g, int r) {
  if constexpr (has_at<G>::value) return g.at(r);
  else return g;
}

// Per-replica strides of a chain's device arguments (elements); the
// scratch arrays always hold nch + 1 entries per replica.
struct ChainStride {
  int64_t s_init = 0;  // the start values
};

constexpr int64_t TWO52 = 1LL << 52;
constexpr int64_t TWO53 = 1LL << 53;
constexpr int64_t SAT = 1LL << 60;
constexpr double SUB_STOP = 1e-14;  // get_d_largest stops once R <= 1e-14
constexpr int CH = 4096;            // chunk length (elements)

struct Map {
  int64_t d0, d1;  // n -> n + (n odd ? d1 : d0)
};

__device__ __forceinline__ Map map_id() { return Map{0, 0}; }
__device__ __forceinline__ int64_t sat(int64_t x) { return x > SAT ? SAT : (x < -SAT ? -SAT : x); }

// f then g
__device__ __forceinline__ Map compose(Map f, Map g) {
  Map r;
  r.d0 = sat(f.d0 + ((f.d0 & 1) ? g.d1 : g.d0));
  r.d1 = sat(f.d1 + ((f.d1 & 1) ? g.d0 : g.d1));
  return r;
}

__device__ __forceinline__ int64_t apply(Map f, int64_t n) { return n + ((n & 1) ? f.d1 : f.d0); }

// binade id b = max(biased exponent, 1); ulp of binade b is 2^(b-1075)
__device__ __forceinline__ int binade_of(double s) {
  const int ef = (int)(((unsigned long long)__double_as_longlong(s) >> 52) & 0x7ff);
  return ef < 1 ? 1 : ef;
}
__device__ __forceinline__ int64_t n_of(double s, int b) {
  return (int64_t)((unsigned long long)__double_as_longlong(s) - ((unsigned long long)(b - 1) << 52));
}
__device__ __forceinline__ double s_of(int b, int64_t n) {
  return __longlong_as_double((long long)(((unsigned long long)(b - 1) << 52) + (unsigned long long)n));
}

// a >= 0 measured in ulps of binade b: q = floor(a/ulp), cls = remainder class
// (0: exact, 1: below half, 2: exactly half, 3: above half).
__device__ __forceinline__ void decomp(double a, int b, int64_t& q, int& cls) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull;
  const int ef = (int)(bits >> 52);
  unsigned long long M = bits & ((1ull << 52) - 1);
  if (ef) M |= 1ull << 52;
  // a running value that is infinite or NaN: finite addends leave it alone,
  // others take the real operation
  if (b >= 2047) { q = ef == 2047 ? SAT : 0; cls = 0; return; }
  const int efp = ef < 1 ? 1 : ef;
  const int shift = b - efp;
  if (shift < 0) { q = SAT; cls = 0; return; }  // a itself is beyond the binade
  if (shift == 0) { q = (int64_t)M; cls = 0; return; }
  if (shift >= 63) { q = 0; cls = M ? 1 : 0; return; }
  q = (int64_t)(M >> shift);
  const unsigned long long r = M & ((1ull << shift) - 1);
  const unsigned long long half = 1ull << (shift - 1);
  cls = r == 0 ? 0 : (r < half ? 1 : (r == half ? 2 : 3));
}

__device__ __forceinline__ Map map_of(int64_t q, int cls, bool sub) {
  const int64_t inc_e = (cls == 3) | ((cls == 2) & (int)(q & 1));
  const int64_t inc_o = (cls == 3) | ((cls == 2) & (int)((q & 1) ^ 1));
  return sub ? Map{-(q + inc_e), -(q + inc_o)} : Map{q + inc_e, q + inc_o};
}

__device__ __forceinline__ Map elem_map(double a, int b, bool sub) {
  int64_t q;
  int cls;
  decomp(a, b, q, cls);
  return map_of(q, cls, sub);
}

// |x| by its bits: fabs is an FP64 instruction
__device__ __forceinline__ double abs_bits(double x) {
  return __longlong_as_double(__double_as_longlong(x) & 0x7fffffffffffffffll);
}

// a >= 0 rounded to units of binade b, where no tie leaves the direction to the
// parity and a is below the binade: the map is then the same for both parities, a
// run's is the sum, and a third of the instructions suffice (they bound every
// pass: the maps of 20 M addends took 105 us at 82% of the integer pipe, the
// sampling pass 280; now 77-91 and 149).
__device__ __forceinline__ bool plain_step(double a, int b, int64_t& r) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(a);
  const int ef = (int)(u >> 52) & 0x7ff;
  const unsigned long long M = (u & 0xfffffffffffffull) | (ef ? 1ull << 52 : 0ull);
  const int shift = b - (ef ? ef : 1) - 1;  // M 2^-shift: halves of a unit
  const int sh = shift < 0 ? 0 : (shift > 63 ? 63 : shift);
  const unsigned long long h = M >> sh;
  r = (int64_t)((h + 1) >> 1);
  return shift >= 0 && !((h & 1) && (h << sh) == M);
}

// One step of the model from n, with exactness check.
__device__ __forceinline__ bool step(int64_t n, double a, int b, bool sub, int64_t& n_out) {
  int64_t q;
  int cls;
  decomp(a, b, q, cls);
  if (!sub) {
    n_out = apply(map_of(q, cls, false), n);
    return n_out <= TWO53;  // result inside binade b, or exactly at its top
  }
  const int64_t lower = b >= 2 ? TWO52 : 0;
  if (q >= SAT || n - q < lower + (cls != 0)) return false;  // exact result leaves binade b
  n_out = apply(map_of(q, cls, true), n);
  return true;
}

// A conservative test that a whole composite step from n0 stayed exact.
__device__ __forceinline__ bool run_valid(int64_t n_end, int b, bool sub) {
  if (!sub) return n_end <= TWO53;
  return n_end >= (b >= 2 ? TWO52 + 1 : 1);
}

// Block-wide exclusive scan of maps in thread order; *total = composite of all.
template <int NT>
__device__ __forceinline__ Map block_excl_scan_map(Map v, Map* smem, Map* total) {
  constexpr int NW = NT / 32;
  Map incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    Map w;
    w.d0 = __shfl_up_sync(0xffffffffu, incl.d0, o);
    w.d1 = __shfl_up_sync(0xffffffffu, incl.d1, o);
    if ((int)lane_id() >= o) incl = compose(w, incl);
  }
  Map wex;
  wex.d0 = __shfl_up_sync(0xffffffffu, incl.d0, 1);
  wex.d1 = __shfl_up_sync(0xffffffffu, incl.d1, 1);
  if (lane_id() == 0) wex = map_id();
  __syncthreads();
  if (lane_id() == 31) smem[warp_id()] = incl;
  __syncthreads();
  // the warp totals, scanned by warp 0 with shuffles: composing them one
  // after another in one thread was most of a round (2 of 4 us at 32 warps)
  if (warp_id() == 0) {
    Map run = (int)lane_id() < NW ? smem[lane_id()] : map_id();
#pragma unroll
    for (int o = 1; o < NW; o <<= 1) {
      Map w;
      w.d0 = __shfl_up_sync(0xffffffffu, run.d0, o);
      w.d1 = __shfl_up_sync(0xffffffffu, run.d1, o);
      if ((int)lane_id() >= o) run = compose(w, run);
    }
    Map ex;
    ex.d0 = __shfl_up_sync(0xffffffffu, run.d0, 1);
    ex.d1 = __shfl_up_sync(0xffffffffu, run.d1, 1);
    if (lane_id() == 0) ex = map_id();
    if ((int)lane_id() < NW) smem[lane_id()] = ex;
    if (lane_id() == NW - 1) smem[NW] = run;
  }
  __syncthreads();
  Map r = compose(smem[warp_id()], wex);
  *total = smem[NW];
  __syncthreads();
  return r;
}

// One segment of a chunk that crosses binades: `map` composes the elements
// between two cuts under binade b (0: none), then the cut element a is added
// for real (unless `last`).
struct Piece {
  Map map;
  double a;
  int b, last;
};
constexpr int PIECES = 64;  // per chunk
constexpr int SLOTS = 32;   // chunks of a chain with pieces: its binade crossings, as a rule
struct Slots {
  Piece p[SLOTS][PIECES];
  int cnt[SLOTS];
};

// Composes s through the pieces of a chunk, checking every prediction;
// `at` (if given) receives {before, after} of each cut, with the segments'
// start values at[j].y of the cut before.
__device__ __forceinline__ bool walk_pieces(const Piece* p, int cnt, double& s, double2* at) {
  double v = s;
  for (int j = 0; j < cnt; ++j) {
    const Piece q = p[j];
    if (q.b) {
      if (binade_of(v) != q.b) return false;
      const int64_t n = apply(q.map, n_of(v, q.b));
      if (!run_valid(n, q.b, false)) return false;
      v = s_of(q.b, n);
    }
    const double before = v;
    if (!q.last) v = __dadd_rn(v, q.a);
    if (at) at[j] = make_double2(before, v);
  }
  s = v;
  return true;
}

struct SplitSmem {
  Piece p[PIECES];
  double2 at[PIECES];
  Map m[33];
  double sum[33];
  int seg[33], cnt[33];  // a segment's binade | CUT once a cut lies in the range
  int ok;
};
constexpr int CUT = 1 << 16, CLASH = 1 << 17;  // CLASH: two binades in one segment

struct Seg {
  Map m;
  int f;  // binade | CUT
  int n;  // cuts
};
__device__ __forceinline__ Seg then(const Seg& x, const Seg& y) {
  Seg r;
  r.m = (y.f & CUT) ? y.m : compose(x.m, y.m);
  const int bx = x.f & 0xffff, by = y.f & 0xffff;
  r.f = (y.f & CUT) ? y.f | (x.f & CLASH)
                    : ((x.f | y.f) & (CUT | CLASH)) | (by ? by : bx) | (bx && by && bx != by ? CLASH : 0);
  r.n = x.n + y.n;
  return r;
}
__device__ __forceinline__ Seg seg_up(const Seg& x, int o) {
  Seg r;
  r.m.d0 = __shfl_up_sync(0xffffffffu, x.m.d0, o);
  r.m.d1 = __shfl_up_sync(0xffffffffu, x.m.d1, o);
  r.f = __shfl_up_sync(0xffffffffu, x.f, o);
  r.n = __shfl_up_sync(0xffffffffu, x.n, o);
  return r;
}

struct ChunkSmem {
  Map maps[33];
  int imin[32];
  double s;
  SplitSmem split;
};

// Exclusive scan of segments in thread order; the whole goes to entry NT / 32 of
// sm's arrays.
template <int NT>
__device__ __forceinline__ Seg block_scan_seg(const Seg& mine, SplitSmem& sm) {
  constexpr int NW = NT / 32;
  const int lane = (int)lane_id(), warp = (int)warp_id();
  Seg inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Seg w = seg_up(inc, o);
    if (lane >= o) inc = then(w, inc);
  }
  Seg wex = seg_up(inc, 1);
  if (lane == 0) wex = Seg{map_id(), 0, 0};
  if (lane == 31) {
    sm.m[warp] = inc.m;
    sm.seg[warp] = inc.f;
    sm.cnt[warp] = inc.n;
  }
  __syncthreads();
  if (warp == 0) {
    Seg run = lane < NW ? Seg{sm.m[lane], sm.seg[lane], sm.cnt[lane]} : Seg{map_id(), 0, 0};
#pragma unroll
    for (int o = 1; o < NW; o <<= 1) {
      const Seg w = seg_up(run, o);
      if (lane >= o) run = then(w, run);
    }
    Seg e = seg_up(run, 1);
    if (lane == 0) e = Seg{map_id(), 0, 0};
    if (lane < NW) {
      sm.m[lane] = e.m;
      sm.seg[lane] = e.f;
      sm.cnt[lane] = e.n;
    }
    if (lane == NW - 1) {
      sm.m[NW] = run.m;
      sm.seg[NW] = run.f;
      sm.cnt[NW] = run.n;
    }
  }
  __syncthreads();
  return then(Seg{sm.m[warp], sm.seg[warp], sm.cnt[warp]}, wex);
}

// Cuts a chunk of additions (element t ITEMS + k at thread t's a[k]) that
// starts at about P0, `slack` units of its last place off at most, and writes
// the pieces to out.  An element is a cut unless the approximate values before
// and after it, slackened, lie in one binade.  Returns the number of pieces (the
// same in every thread), 0 if they are more than PIECES.  pre: the composite
// before the thread's first element, in the segment pre.n; cuts: the thread's
// cut elements, as bits.  Integer comparisons of the bit patterns: GB300 adds
// 2 FP64 numbers per SM and clock.  Bound by its dependent steps: ~25 us, where a
// round per crossing (scan, search, one addition) took 4-9 us each and a first
// chunk has a dozen (compressing o10v40's 160000 elements: the two walks 319 ->
// 28 us, the sampling pass 130 -> 37, the chunk maps 17 -> 41).
template <int NT, int ITEMS>
__device__ __forceinline__ int split_chunk(const double* a, int n_in, double P0, int64_t slack, SplitSmem& sm, Piece* out,
                                           Seg& pre, unsigned& cuts) {
  constexpr int NW = NT / 32;
  const int t = threadIdx.x, lane = (int)lane_id(), warp = (int)warp_id();
  double loc = 0.0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) loc += a[k];  // (zeros past n_in)
  double incl = loc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double w = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += w;
  }
  double ex = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane == 0) ex = 0.0;
  __syncthreads();
  if (lane == 31) sm.sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    double run = lane < NW ? sm.sum[lane] : 0.0;
#pragma unroll
    for (int o = 1; o < NW; o <<= 1) {
      const double w = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += w;
    }
    double e = __shfl_up_sync(0xffffffffu, run, 1);
    if (lane == 0) e = 0.0;
    if (lane < NW) sm.sum[lane] = e;
  }
  __syncthreads();
  const double P = P0 + (sm.sum[warp] + ex);
  auto binade = [&](double p, double q, int& b) {  // false: a cut
    const long long lo = __double_as_longlong(p) - slack, hi = __double_as_longlong(q) + slack;
    if (!(q < 1e300)) return false;  // (NaN too)
    const int bl = lo < 0 ? 0 : (int)(lo >> 52), bh = (int)(hi >> 52);
    b = bl < 1 ? 1 : bl;
    return b == (bh < 1 ? 1 : bh);
  };
  Seg mine{map_id(), 0, 0};
  cuts = 0;
  double p = P;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    if (t * ITEMS + k < n_in) {
      const double q = p + a[k];
      int b;
      if (binade(p, q, b)) {
        mine.m = compose(mine.m, elem_map(a[k], b, false));
        mine.f = (mine.f & CUT) | b;
      } else {
        cuts |= 1u << k;
        mine.m = map_id();
        mine.f = CUT;
        ++mine.n;
      }
      p = q;
    }
  }
  pre = block_scan_seg<NT>(mine, sm);
  const int total = sm.cnt[NW] + 1;
  if (total > PIECES || (sm.seg[NW] & CLASH)) return 0;
  if (cuts) {
    Map m = pre.m;
    int f = pre.f & 0xffff, j = pre.n;
    p = P;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      if (t * ITEMS + k < n_in) {
        const double q = p + a[k];
        if ((cuts >> k) & 1u) {
          out[j++] = Piece{m, a[k], f, 0};
          m = map_id();
          f = 0;
        } else {
          int b;
          binade(p, q, b);
          m = compose(m, elem_map(a[k], b, false));
          f = b;
        }
        p = q;
      }
    }
  }
  if (t == 0) out[total - 1] = Piece{sm.m[NW], 0.0, sm.seg[NW] & 0xffff, 1};
  return total;
}

struct ConsNull {
  __device__ __forceinline__ void operator()(int64_t, double, double, double) const {}
};

// A consumer with a method finish() is told once per thread, after the
// thread's last element (so it can keep a per-thread result and publish it
// with one atomic per warp).
template <class C, class = void>
struct has_finish : std::false_type {};
template <class C>
struct has_finish<C, std::void_t<decltype(std::declval<C&>().finish())>> : std::true_type {};

// A consumer that only looks for values the running sum passes has start(s), the
// state at a thread's first element, and step(state, i, s), the sum after element i
// (repeated past the chunk's end); runs() says whether they can be used.
template <class C, class = void>
struct has_run : std::false_type {};
template <class C>
struct has_run<C, std::void_t<decltype(std::declval<const C&>().runs())>> : std::true_type {};

// A chain's length: n elements, or (dev) the count at dev[rep * stride],
// never above n; nothing at all where the word skip[rep * sstride] is set.
struct Len {
  int64_t n = 0;
  const int64_t* dev = nullptr;
  int64_t stride = 0;
  const int* skip = nullptr;
  int64_t sstride = 0;
  __device__ __forceinline__ int64_t get(int rep) const {
    if (skip && skip[rep * sstride]) return 0;
    if (!dev) return n;
    const int64_t d = dev[rep * stride];
    return d < n ? d : n;
  }
};

// Exact processing of one chunk by the whole block.  Thread t owns the
// contiguous elements [t*ITEMS, t*ITEMS+ITEMS).  cons(i, before, after, a)
// is called once for every element, in no particular order.  Returns the
// exact running value after the chunk (the same in every thread).
template <int NT, int ITEMS, class Gen, class Cons>
__device__ double block_exact_chunk(const Gen& gen, int64_t base, int n_in, double s_start, bool sub,
                                    Cons& cons, ChunkSmem& sm) {
  double a[ITEMS];
  const int t = threadIdx.x;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int i = t * ITEMS + k;
    a[k] = i < n_in ? gen(base + i) : 0.0;
  }
  double s = s_start;
  int p = 0;
  for (int round = 0; round <= NT * ITEMS && p < n_in; ++round) {
    if (sub && !(s > SUB_STOP)) {  // the remaining-norm chain is over: R stays put
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        const int i = t * ITEMS + k;
        if (i >= p && i < n_in) cons(base + i, s, s, a[k]);
      }
      p = n_in;
      break;
    }
    const int b = binade_of(s);
    const int64_t n0 = n_of(s, b);
    bool plain = b < 2047;
    int64_t sum = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const int i = t * ITEMS + k;
      int64_t r;
      plain &= plain_step(i >= p ? a[k] : 0.0, b, r);  // (zeros past n_in)
      sum += r;
    }
    if (sub) sum = -sum;
    Map agg{sum, sum};
    if (!plain) {
      agg = map_id();
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        const int i = t * ITEMS + k;
        if (i >= p && i < n_in) agg = compose(agg, elem_map(a[k], b, sub));
      }
    }
    Map tot;
    const Map pre = block_excl_scan_map<NT>(agg, sm.maps, &tot);
    int64_t n = apply(pre, n0);
    int first_bad = INT_MAX;
    int64_t n_bad = 0;
    int k_bad = 0;
    int istar = INT_MAX;
    // the running value is monotone, so when the run's end is still inside
    // the binade every step is: the search for the step that leaves it (a
    // second pass over the items and a block minimum) runs only otherwise
    if (!run_valid(apply(tot, n0), b, sub)) {
      if (!sub && round == 0) {
        // all crossings at once: the rounds below take one each (4-9 us; the
        // first chunk of a chain has a dozen)
        Seg seg;
        unsigned cuts;
        const int cnt = split_chunk<NT, ITEMS>(a, n_in, s, 256 + n_in, sm.split, sm.split.p, seg, cuts);
        __syncthreads();
        if (t == 0) {
          double v = s;
          sm.split.ok = cnt > 0 && walk_pieces(sm.split.p, cnt, v, sm.split.at);
          sm.s = v;
        }
        __syncthreads();
        if (sm.split.ok) {
          int j = seg.n, bj = sm.split.p[j].b;
          const double s0 = j ? sm.split.at[j - 1].y : s;
          int64_t nj = bj ? apply(seg.m, n_of(s0, bj)) : 0;
#pragma unroll
          for (int k = 0; k < ITEMS; ++k) {
            const int i = t * ITEMS + k;
            if (i < n_in) {
              if ((cuts >> k) & 1u) {
                const double2 v = sm.split.at[j];
                cons(base + i, v.x, v.y, a[k]);
                bj = sm.split.p[++j].b;
                nj = n_of(v.y, bj);
              } else {
                const int64_t nn = apply(elem_map(a[k], bj, false), nj);
                cons(base + i, s_of(bj, nj), s_of(bj, nn), a[k]);
                nj = nn;
              }
            }
          }
          return sm.s;
        }
      }
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        const int i = t * ITEMS + k;
        if (i >= p && i < n_in && first_bad == INT_MAX) {
          int64_t nn;
          if (step(n, a[k], b, sub, nn)) {
            n = nn;
          } else {
            first_bad = i;
            n_bad = n;
            k_bad = k;
          }
        }
      }
      istar = block_min<int>(first_bad, sm.imin);
      n = apply(pre, n0);
    }
    bool done = false;
    if constexpr (has_run<Cons>::value) {
      if (plain && istar == INT_MAX && cons.runs()) {
        auto run = cons.start(s_of(b, n));
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
          const int i = t * ITEMS + k;
          int64_t r;
          plain_step(i >= p ? a[k] : 0.0, b, r);
          n += sub ? -r : r;
          cons.step(run, base + i, s_of(b, n));
        }
        done = true;
      }
    }
    if (!done) {
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        const int i = t * ITEMS + k;
        if (i >= p && i < n_in && i < istar) {
          int64_t nn;
          step(n, a[k], b, sub, nn);
          cons(base + i, s_of(b, n), s_of(b, nn), a[k]);
          n = nn;
        }
      }
    }
    if (istar == INT_MAX) {
      s = s_of(b, apply(tot, n0));
      p = n_in;
      break;
    }
    if (first_bad == istar) {
      const double sb = s_of(b, n_bad);
      const double sa = sub ? __dsub_rn(sb, a[k_bad]) : __dadd_rn(sb, a[k_bad]);
      cons(base + istar, sb, sa, a[k_bad]);
      sm.s = sa;
    }
    __syncthreads();
    s = sm.s;
    p = istar + 1;
    __syncthreads();
  }
  return s;
}

// ---------------------------------------------------------------- kernels

// K_A: approximate sum of each chunk (fixed reduction tree).
template <class Gen>
__global__ void __launch_bounds__(256) k_chunk_sums(Gen gen0, Len ln, double* csum) {
  const int rep = blockIdx.y;
  const int64_t len = ln.get(rep);
  const int64_t base = (int64_t)blockIdx.x * CH;
  if (base >= len) return;
  const Gen gen = replica_of(gen0, rep);
  csum += (int64_t)rep * (fricc_cdiv(ln.n, CH) + 1);
  __shared__ double red[32];
  double acc = 0.0;
  for (int r = 0; r < CH / 256; ++r) {
    const int64_t i = base + r * 256 + threadIdx.x;
    if (i < len) acc += gen(i);
  }
  const double tot = block_sum_det(acc, red);
  if (threadIdx.x == 0) csum[blockIdx.x] = tot;
}

// K_B (one block of 1024): approximate prefix of the chunk sums and the
// per-chunk binade prediction: cbin[c] = binade if clean; else minus the slot
// for its pieces, counted from 1 (0: none left, or a chain of subtractions), and
// csum[c] becomes the approximate value at the chunk's start.  The
// prefix is a shuffle scan: one thread adding 1024 partials (dependent FP64
// additions, ~55 ns each on this part) took 58 us a call, three calls a
// compression; now 4-5 us.
static __global__ void __launch_bounds__(1024) k_classify(double* csum, Len ln, const double* s_init_dev,
                                                   int sub, int* cbin, ChainStride cs) {
  const int rep = blockIdx.x;
  const int64_t nch = fricc_cdiv(ln.get(rep), CH), cap = fricc_cdiv(ln.n, CH) + 1;
  csum += (int64_t)rep * cap;
  cbin += (int64_t)rep * cap;
  const double s_init = s_init_dev[rep * cs.s_init];
  __shared__ double wtot[33];
  __shared__ int used;
  if (threadIdx.x == 0) used = 0;
  const int64_t per = fricc_cdiv(nch, 1024);
  const int64_t c0 = threadIdx.x * per;
  const int64_t c1 = c0 + per < nch ? c0 + per : nch;
  double loc = 0.0;
  for (int64_t c = c0; c < c1; ++c) loc += csum[c];
  double incl = loc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double w = __shfl_up_sync(0xffffffffu, incl, o);
    if ((int)lane_id() >= o) incl += w;
  }
  double excl = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane_id() == 0) excl = 0.0;
  if (lane_id() == 31) wtot[warp_id()] = incl;
  __syncthreads();
  if (warp_id() == 0) {
    double run = wtot[lane_id()];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double w = __shfl_up_sync(0xffffffffu, run, o);
      if ((int)lane_id() >= o) run += w;
    }
    double ex = __shfl_up_sync(0xffffffffu, run, 1);
    if (lane_id() == 0) ex = 0.0;
    wtot[lane_id()] = ex;
    if (lane_id() == 31) wtot[32] = run;
  }
  __syncthreads();
  const double scale = fabs(s_init) + wtot[32];
  double pre = wtot[warp_id()] + excl;
  for (int64_t c = c0; c < c1; ++c) {
    const double P0 = sub ? s_init - pre : s_init + pre;
    pre += csum[c];
    const double P1 = sub ? s_init - pre : s_init + pre;
    const double margin = scale * ((double)(c + 1) * CH * 0x1p-50 + 0x1p-44);
    const double lo = (sub ? P1 : P0) - margin;
    const double hi = (sub ? P0 : P1) + margin;
    int b = 0;
    if (lo > (sub ? SUB_STOP : 0.0) && hi < 1e300) {
      const int b_lo = binade_of(lo), b_hi = binade_of(hi);
      if (b_lo == b_hi) b = b_lo;
    }
    if (b == 0 && !sub) {
      const int k = atomicAdd(&used, 1);
      if (k < SLOTS) b = -(k + 1);
      csum[c] = P0;
    }
    cbin[c] = b;
  }
}

// K_C: composite map of each clean chunk under its predicted binade; the
// pieces of the others.
template <class Gen>
__global__ void __launch_bounds__(256) k_chunk_maps(Gen gen0, Len ln, int sub, const int* cbin, Map* cmap,
                                                    const double* csum, Slots* slots) {
  constexpr int NT = 256, ITEMS = CH / NT;
  const int rep = blockIdx.y;
  const int64_t len = ln.get(rep);
  const int64_t base = (int64_t)blockIdx.x * CH;
  if (base >= len) return;
  const Gen gen = replica_of(gen0, rep);
  const int64_t cap = fricc_cdiv(ln.n, CH) + 1;
  cbin += (int64_t)rep * cap;
  cmap += (int64_t)rep * cap;
  __shared__ Map smaps[33];
  __shared__ SplitSmem ssm;
  const int b = cbin[blockIdx.x];
  if (b == 0) return;  // uniform per block
  const int n_in = (int)(len - base < CH ? len - base : CH);
  double a[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const int i = threadIdx.x * ITEMS + k;
    a[k] = i < n_in ? gen(base + i) : 0.0;
  }
  if (b < 0) {
    Seg pre;
    unsigned cuts;
    slots += rep;
    // the chain's own rounding: half a unit per element; the prediction's: a
    // unit per addition of its trees
    const int cnt = split_chunk<NT, ITEMS>(a, n_in, csum[rep * cap + blockIdx.x], base + n_in + cap / 256 + 256, ssm,
                                           slots->p[-b - 1], pre, cuts);
    if (threadIdx.x == 0) slots->cnt[-b - 1] = cnt;
    return;
  }
  bool plain = true;
  int64_t sum = 0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    int64_t r;
    plain &= plain_step(a[k], b, r);
    sum += r;
  }
  if (sub) sum = -sum;
  Map agg{sum, sum};
  if (!plain) {
    agg = map_id();
#pragma unroll 1
    for (int k = 0; k < ITEMS; ++k) {
      const int64_t i = base + threadIdx.x * ITEMS + k;
      if (i < len) agg = compose(agg, elem_map(gen(i), b, sub != 0));
    }
  }
  Map tot;
  block_excl_scan_map<NT>(agg, smaps, &tot);
  if (threadIdx.x == 0) cmap[blockIdx.x] = tot;
}

// K_D (one block of 1024): the exact chain over chunks.  cstart[c] receives
// the exact running value at the start of chunk c, cstart[nch] the total,
// which also goes to *end (if given).  The loop over runs of chunks takes the
// chains of subtractions, and an addition's from where a prediction fails.
constexpr int WALK_Q = 256;  // pieces of all cut chunks
template <class Gen>
__global__ void __launch_bounds__(1024) k_walk(Gen gen0, Len ln, const double* s_init_dev, int sub,
                                               const int* cbin, const Map* cmap, const Slots* slots, double* cstart,
                                               double* end, int64_t end_stride, ChainStride cs) {
  const int rep = blockIdx.x;
  const int64_t len = ln.get(rep);
  const Gen gen = replica_of(gen0, rep);
  {
    const int64_t st = (int64_t)rep * (fricc_cdiv(ln.n, CH) + 1);
    cbin += st;
    cmap += st;
    cstart += st;
    slots += rep;
  }
  const double s_init = s_init_dev[rep * cs.s_init];
  constexpr int NT = 1024;
  __shared__ Map smaps[33];
  __shared__ int simin[32];
  __shared__ ChunkSmem csm;
  __shared__ Piece q[WALK_Q];
  __shared__ int64_t cut[PIECES], cfail;
  __shared__ int off[SLOTS + 1];
  const int64_t nch = fricc_cdiv(len, CH);
  double s = s_init;
  int64_t c = 0;
  if (!sub) {  // all chunks at once: the segments between the cut ones by a scan, then one thread
    SplitSmem& sm = csm.split;
    const int64_t per = fricc_cdiv(nch, NT), c0 = threadIdx.x * per, c1 = c0 + per < nch ? c0 + per : nch;
    Seg mine{map_id(), 0, 0};
    for (int64_t k = c0; k < c1; ++k) {
      const int b = cbin[k];
      mine = then(mine, b > 0 ? Seg{cmap[k], b, 0} : Seg{map_id(), CUT, 1});
    }
    const Seg pre = block_scan_seg<NT>(mine, sm);
    const int ncut = sm.cnt[NT / 32];
    if (ncut < PIECES && !(sm.seg[NT / 32] & CLASH)) {
      Seg at = pre;
      for (int64_t k = c0; k < c1; ++k) {
        const int b = cbin[k];
        if (b <= 0) {
          sm.p[at.n] = Piece{at.m, 0.0, at.f & 0xffff, 0};
          cut[at.n] = k;
        }
        at = then(at, b > 0 ? Seg{cmap[k], b, 0} : Seg{map_id(), CUT, 1});
      }
      if (threadIdx.x == 0) sm.p[ncut] = Piece{sm.m[NT / 32], 0.0, sm.seg[NT / 32] & 0xffff, 1};
      // the cut chunks' pieces, slot by slot: a warp each
      const int slot = (int)warp_id(), used = ncut < SLOTS ? ncut : SLOTS;
      if (threadIdx.x < 32) {
        const int v = (int)threadIdx.x < used ? slots->cnt[threadIdx.x] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int w = __shfl_up_sync(0xffffffffu, incl, o);
          if ((int)threadIdx.x >= o) incl += w;
        }
        off[threadIdx.x + 1] = incl;
        if (threadIdx.x == 0) off[0] = 0;
      }
      __syncthreads();
      for (int k = (int)lane_id(); k < off[slot + 1] - off[slot]; k += 32)
        if (off[slot] + k < WALK_Q) q[off[slot] + k] = slots->p[slot][k];
      __syncthreads();
      if (threadIdx.x == 0) {
        double v = s;
        int64_t fail = nch;
        for (int j = 0; j <= ncut; ++j) {
          const int64_t first = j ? cut[j - 1] + 1 : 0;
          const double before = v;
          if (!walk_pieces(&sm.p[j], 1, v, nullptr)) {  // (its real addition is of zero)
            fail = first;
            v = before;
            break;
          }
          sm.at[j] = make_double2(before, v);
          if (j == ncut) break;
          const int k = -cbin[cut[j]] - 1, o = k >= 0 ? off[k] : 0, cnt = k >= 0 ? off[k + 1] - o : 0;
          const double at_cut = v;
          if (cnt == 0 || o + cnt > WALK_Q || !walk_pieces(q + o, cnt, v, nullptr)) {
            fail = cut[j];
            v = at_cut;
            break;
          }
        }
        cfail = fail;
        csm.s = v;
      }
      __syncthreads();
      at = pre;
      for (int64_t k = c0; k < c1 && k < cfail; ++k) {
        const int b = cbin[k];
        cstart[k] = b > 0 ? s_of(b, apply(at.m, n_of(sm.at[at.n].x, b))) : sm.at[at.n].y;
        at = then(at, b > 0 ? Seg{cmap[k], b, 0} : Seg{map_id(), CUT, 1});
      }
      s = csm.s;
      c = cfail;
      __syncthreads();
    }
  }
  for (int64_t guard = 0; guard <= 2 * nch && c < nch; ++guard) {
    if (sub && !(s > SUB_STOP)) break;
    const int b = binade_of(s);
    const int64_t n0 = n_of(s, b);
    const int64_t ct = c + threadIdx.x;
    const bool ok = ct < nch && cbin[ct] == b;
    const int L = block_min<int>(ok ? INT_MAX : (int)threadIdx.x, simin);
    if (L > 0) {
      const Map mine = (ok && (int)threadIdx.x < L) ? cmap[ct] : map_id();
      Map tot;
      const Map pre = block_excl_scan_map<NT>(mine, smaps, &tot);
      const Map incl = compose(pre, mine);
      const int64_t n_end = apply(incl, n0);
      const bool bad = (int)threadIdx.x < L && !run_valid(n_end, b, sub != 0);
      int J = block_min<int>(bad ? (int)threadIdx.x : INT_MAX, simin);
      if (J > L) J = L;
      if (J > NT) J = NT;
      if ((int)threadIdx.x < J) cstart[ct] = s_of(b, apply(pre, n0));
      if (J > 0) {
        // the thread J-1 holds the end value; every thread can recompute it
        // from the block data only through smem, so pass it along.
        if ((int)threadIdx.x == J - 1) csm.s = s_of(b, n_end);
        __syncthreads();
        s = csm.s;
        __syncthreads();
        c += J;
        continue;
      }
    }
    if (threadIdx.x == 0) cstart[c] = s;
    const int64_t base = c * CH;
    const int n_in = (int)(len - base < CH ? len - base : CH);
    ConsNull none;
    s = block_exact_chunk<NT, CH / NT>(gen, base, n_in, s, sub != 0, none, csm);
    c += 1;
  }
  // chunks after an exhausted remaining-norm chain keep the final value
  for (int64_t cc = c + threadIdx.x; cc < nch; cc += NT) cstart[cc] = s;
  if (threadIdx.x == 0) {
    cstart[nch] = s;
    if (end) end[rep * end_stride] = s;
  }
}

// K_E: every element's exact before/after values, from the exact chunk starts.
template <class Gen, class Cons>
__global__ void __launch_bounds__(512) k_emit(Gen gen0, Cons cons0, Len ln, int sub, const double* cstart) {
  constexpr int NT = 512;
  const int rep = blockIdx.y;
  const int64_t len = ln.get(rep);
  const int64_t base = (int64_t)blockIdx.x * CH;
  if (base >= len) return;
  const Gen gen = replica_of(gen0, rep);
  Cons cons = replica_of(cons0, rep);
  cstart += (int64_t)rep * (fricc_cdiv(ln.n, CH) + 1);
  __shared__ ChunkSmem csm;
  const int n_in = (int)(len - base < CH ? len - base : CH);
  block_exact_chunk<NT, CH / NT>(gen, base, n_in, cstart[blockIdx.x], sub != 0, cons, csm);
  if constexpr (has_finish<Cons>::value) cons.finish();
}

struct ChainScratch {
  double* csum = nullptr;
  int* cbin = nullptr;
  Map* cmap = nullptr;
  double* cstart = nullptr;
  Slots* slots = nullptr;  // one per replica
  int64_t cap = 0;
  int reps = 0;
};

// Runs the chain over gen(0..len-1) from s_init.  On return (stream order)
// scratch.cstart[nch] holds the exact final value, which also goes to *end
// (device, end_stride doubles per replica) when given; with EMIT, cons has
// seen every element.  have_sums: sc.csum already holds the chunk sums (a
// kernel that made the addends summed them in the same pass).
inline int chain_scratch(ChainScratch& sc, int64_t entries, cudaStream_t st, int reps = 1) {
  if (sc.reps < reps) {
    fricc_free(sc.slots, st);
    sc.reps = 0;
    if (int rc = fricc_alloc_t(&sc.slots, reps, st)) return rc;
    sc.reps = reps;
  }
  if (sc.cap >= entries) return FRICC_OK;
  fricc_free(sc.csum, st);
  fricc_free(sc.cbin, st);
  fricc_free(sc.cmap, st);
  fricc_free(sc.cstart, st);
  int rc = fricc_alloc_t(&sc.csum, entries, st);
  if (!rc) rc = fricc_alloc_t(&sc.cbin, entries, st);
  if (!rc) rc = fricc_alloc_t(&sc.cmap, entries, st);
  if (!rc) rc = fricc_alloc_t(&sc.cstart, entries, st);
  if (!rc) sc.cap = entries;
  return rc;
}

template <class Gen, class Cons, bool EMIT>
int run_chain(const Gen& gen, const Len& len, const double* s_init_dev, bool sub, const Cons& cons,
              ChainScratch& sc, cudaStream_t st, int R = 1, ChainStride cs = ChainStride{}, bool have_sums = false,
              double* end = nullptr, int64_t end_stride = 0) {
  const int64_t nch = fricc_cdiv(len.n, CH);
  if (nch > INT_MAX / 2 || R < 1 || R > 65535) return FRICC_ERR_ARG;
  if (R > 1) {  // the batch's scratch: nch + 1 entries per replica, sized by the caller
    if (sc.cap < R * (nch + 1) || sc.reps < R) return FRICC_ERR_ARG;
    if (nch == 0) return FRICC_ERR_ARG;
  } else if (int rc = chain_scratch(sc, nch + 1, st)) {
    return rc;
  }
  if (nch == 0) {
    FRICC_CUDA(cudaMemcpyAsync(sc.cstart, s_init_dev, sizeof(double), cudaMemcpyDeviceToDevice, st));
    if (end) FRICC_CUDA(cudaMemcpyAsync(end, s_init_dev, sizeof(double), cudaMemcpyDeviceToDevice, st));
    return FRICC_OK;
  }
  const dim3 gch((unsigned)nch, (unsigned)R);
  if (!have_sums) k_chunk_sums<Gen><<<gch, 256, 0, st>>>(gen, len, sc.csum);
  k_classify<<<R, 1024, 0, st>>>(sc.csum, len, s_init_dev, sub ? 1 : 0, sc.cbin, cs);
  k_chunk_maps<Gen><<<gch, 256, 0, st>>>(gen, len, sub ? 1 : 0, sc.cbin, sc.cmap, sc.csum, sc.slots);
  k_walk<Gen><<<R, 1024, 0, st>>>(gen, len, s_init_dev, sub ? 1 : 0, sc.cbin, sc.cmap, sc.slots, sc.cstart, end,
                                  end_stride, cs);
  if (EMIT) k_emit<Gen, Cons><<<gch, 512, 0, st>>>(gen, cons, len, sub ? 1 : 0, sc.cstart);
  fricc_note_launch(3 + (have_sums ? 0 : 1) + (EMIT ? 1 : 0));
  FRICC_LAUNCH_CHECK();
  return FRICC_OK;
}

inline void free_chain(ChainScratch& sc, cudaStream_t st) {
  fricc_free(sc.csum, st);
  fricc_free(sc.cbin, st);
  fricc_free(sc.cmap, st);
  fricc_free(sc.cstart, st);
  fricc_free(sc.slots, st);
  sc = ChainScratch{};
}

}  // namespace exact
