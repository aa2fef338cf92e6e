// FP64-accurate GEMM on the tcgen05 tensor cores, by modular integer arithmetic.
//
// GB300 runs FP64 FMA at 2 per SM per clock (1.26 TFLOP/s) and BF16 tensor
// products at ~1.9 PFLOP/s.  A product of two FP64 matrices is computed here
// exactly, as integers, from 15 BF16 products (the residue-number form of
// Ozaki's splitting: Ozaki, Uchino, Imamura 2024-25):
//
// * each row x of an operand is scaled by a power of two to integers
//   X = rint(x 2^s) with 2^60 < |X|_2 <= 2^61 (one shift per row), and X is
//   reduced modulo 15 pairwise coprime odd moduli <= 361 to balanced residues,
//   integers of at most 180: exact in BF16.  Each modulus is one operand
//   "plane";
// * one persistent tcgen05 kernel multiplies the planes, modulus by modulus:
//   512 products of at most 180^2 sum to less than 2^24, so FP32 accumulation
//   in tensor memory is exact over 512 k; the epilogue warps drain it every
//   512 k and reduce it modulo p in FP32 into registers.  (14 moduli up to 512
//   need a drain every 256 k and were no faster: the drains, not the MMAs,
//   set the pace.)
// * by Cauchy-Schwarz |sum X Y| <= 2^122, below an eighth of the product of
//   the moduli (2^125.6), so the 15 residues determine it: the Chinese
//   remainder sum is taken as a 96-bit binary fraction of that product (it
//   wraps by itself) and rounded once to FP64.
//
// The only error is the rounding of X: 0.29 per element against row norms
// of 2^60.5, i.e. 2^-62 |x||y| in an output, where an FP64 FMA chain of n
// terms commits about 0.2 n^1/2 2^-53 (sum x^2 y^2)^1/2.  The two part where
// the large elements of x meet the small ones of y, so a 16th plane holds the
// squares (BF16): every output is checked against n s2 >= 2^-16 |x|^2 |y|^2, s2
// the largest sum x^2 y^2 of a run of 512 k, and one that fails (true zeros
// apart: ZERO_SPAN), that belongs to a row that is not finite, or whose pipeline
// gave up, is recomputed with FP64 FMAs (k_mod_fix).  (At that line, where all
// squares sit in one run, the error is two to three times one chain's, and by the
// root of its slices more against the FP64 kernel's split sums; from 2^-14 up it
// is below a chain's.  A line at 2^-13 listed 70 tiles an o30v150 iteration, 0.9
// ms, and changed no measured error; 2^-12 took 56 ms.)
// A result is the same in any tiling, batch or split of K: integer sums do not
// depend on their order, a sum has one balanced residue whatever the order of its
// reductions (make_tab), and the check compares the largest of the runs' squares,
// which are the same runs in every split.  (With one of the moduli even, slices'
// residues summed without a reduction and their squares added, the fraction's
// rounding and the check's outcome followed the split, and so the batch.)
//
// Measured on a GB300 (operands prepared; DFMA kernel): 900 x 22500 x 22500
// 9.1 ms; 4500^3 2.05 ms (152 ms); 2000^3 0.26 ms (14.0 ms); 400^3 30 us
// (279 us); 675000 x 30 x 150 0.97 ms (5.25 ms).  Converting an operand: 10-11 ps
// an element.  Error (2-norm, against 64 bits) of the o30v150 iteration over
// several inputs: 7.0e-16 to 1.6e-15, 2.3e-15 on the FP64 pipe.
#include <climits>

#include "gemm_mod.cuh"
#include "tc.cuh"

namespace mod {

using namespace tc;

constexpr int NP = 15;        // moduli
constexpr int PLANES = NP + 1;  // + the squares
constexpr int MEW = 16;       // epilogue warps: four per TMEM lane quadrant, each a quarter of the columns
constexpr int MNT = 32 * (2 + MEW);
constexpr int KC = 8;         // 64-wide K blocks per exact FP32 run (512 k)
constexpr int64_t MAX_K = 1ll << 22;
constexpr int MAX_KS = 64;    // K slices; their residues are summed in 32 bits

struct Tab {
  int p[NP] = {};
  int c[NP][3] = {};   // 2^(16 (j+1)) mod p, balanced
  int f[NP][3] = {};   // round(2^96 y / p) in signed 32-bit limbs, y = (M/p)^-1 mod p
  unsigned long long mtop = 0;  // M >> 62, in [2^63, 2^64)
};

// The moduli are odd, and their FP32 reciprocals close enough that x - p rint(x
// fl(1/p)) is the residue in (-p/2, p/2) for every |x| of a run (canonical()):
// with 360, 349 or 343 a residue next to half of p could come out on either side,
// depending on the run it was reduced in.
constexpr bool canonical(int p) {
  const int h = (p - 1) / 2;
  const double e = (double)(1.0f / (float)p) * p - 1.0;  // exact
  return p % 2 == 1 && 2.0 * (e < 0 ? -e : e) * (512.0 * h * h + h) < 1.0;
}

constexpr Tab make_tab() {
  Tab t;
  const int p[NP] = {361, 359, 353, 347, 341, 339, 337, 335, 331, 329, 317, 313, 311, 307, 299};
  unsigned __int128 M = 1;
  for (int i = 0; i < NP; ++i) {
    t.p[i] = p[i];
    M *= (unsigned)p[i];
  }
  t.mtop = (unsigned long long)(M >> 62);
  for (int i = 0; i < NP; ++i) {
    int w = 1;
    for (int j = 0; j < 3; ++j) {
      for (int b = 0; b < 16; ++b) w = 2 * w % p[i];
      t.c[i][j] = 2 * w > p[i] ? w - p[i] : w;
    }
    const int q = (int)((M / (unsigned)p[i]) % (unsigned)p[i]);
    int y = 1;
    while (q * y % p[i] != 1) ++y;
    const unsigned __int128 num = ((unsigned __int128)y << 96);
    unsigned __int128 f = (num + (unsigned)p[i] / 2) / (unsigned)p[i];
    for (int l = 0; l < 3; ++l) {
      const unsigned lo = (unsigned)f;
      const long long s = lo >= 0x80000000u ? (long long)lo - (1ll << 32) : (long long)lo;
      t.f[i][l] = (int)s;
      f = (f >> 32) + (lo >= 0x80000000u ? 1u : 0u);
    }
  }
  return t;
}
__device__ constexpr Tab TAB = make_tab();
static_assert((TAB.mtop >> 63) == 1, "the product of the moduli lies in [2^125, 2^126)");
constexpr bool moduli_hold() {
  for (int i = 0; i < NP; ++i) {
    if (!canonical(make_tab().p[i])) return false;
    for (int j = 0; j < i; ++j) {
      int a = make_tab().p[i], b = make_tab().p[j];
      while (b) {
        const int r = a % b;
        a = b;
        b = r;
      }
      if (a != 1) return false;
    }
  }
  return true;
}
static_assert(moduli_hold(), "pairwise coprime moduli with one balanced residue");

__constant__ float c_p[NP] = {361, 359, 353, 347, 341, 339, 337, 335, 331, 329, 317, 313, 311, 307, 299};

constexpr float MAGIC = 12582912.0f;  // 1.5 * 2^23: adding it rounds a float to an integer

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 upk2(f32x2 r) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(r));
  return f;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// x - p rint(x / p) for integer-valued |x| <= 2^24: exact
__device__ __forceinline__ f32x2 reduce2(f32x2 x, f32x2 inv, f32x2 negp) {
  const f32x2 q = add2(fma2(x, inv, pk2(MAGIC, MAGIC)), pk2(-MAGIC, -MAGIC));
  return fma2(q, negp, x);
}

// ------------------------------------------------------------ operands
// Buffer of an operand: int sh[rows], unsigned cnt[rows] (nonzeros, and in the
// top byte the row's span, below), then at a 1 KB boundary the planes, [PLANES][nkb][rows][64] BF16 (K padded with
// zeros to whole 64-wide blocks).  K-blocked, so that a TMA box of 256 rows is one
// run of 32 KB and the conversion's stores are runs of 4 KB: with plain
// K-major rows (45 KB apart at K = 22500) both missed the TLB on every row
// (the (ac|bd) block of o30v150 converted in 17.2 ms, its product at 815 TFLOP/s).
struct Layout {
  int64_t rows, nkb, off_cnt, off_planes, bytes;
};
__host__ inline Layout layout(int64_t rows, int64_t k) {
  Layout l;
  l.rows = rows;
  l.nkb = (k + BK - 1) / BK;
  l.off_cnt = rows * 4;
  l.off_planes = (rows * 8 + 1023) / 1024 * 1024;
  l.bytes = l.off_planes + (int64_t)PLANES * l.nkb * rows * (BK * 2);
  return l;
}
constexpr int SH_BAD = INT_MIN;  // a row with an infinity or a NaN

// a contraction index of two levels costs a division, which must not run
// (predicated off) where there is one
template <bool K2>
__device__ __forceinline__ int64_t koff(const ModView& v, int64_t k) {
  if constexpr (K2) return v.kat(k);
  else return k * v.sk;
}

// A row's (or a part of a row's) largest biased exponent (0: all zero), its
// nonzeros' number and smallest exponent less 1 (all ones: none), and the sum of
// (|x| 2^(1023 - emax))^2 in units of 2^-28, rounded up.
struct RowStat {
  unsigned long long sum;
  int emax;
  unsigned short cnt, low;  // (of at most SCH elements)
};
constexpr int SCH = 256;  // k of one part: a thread's share stays in registers

__device__ __forceinline__ int exp_of(unsigned long long u) {  // biased, subnormals as 1, zero as 0
  const int e = (int)((u >> 52) & 0x7ff);
  return e ? e : ((u << 1) ? 1 : 0);
}

__device__ __forceinline__ unsigned sq_units(unsigned long long u, int emax) {
  const int e = exp_of(u);
  if (e == 0) return 0u;
  if (emax - e > 15) return 1u;
  const unsigned long long m = (u & 0xfffffffffffffull) | ((u >> 52) & 0x7ff ? 1ull << 52 : 0ull);
  // |x| 2^(1023 - emax) rounded up, in [0, 2]
  const float v = __fmul_ru((float)((unsigned)(m >> 29) + 1u), __uint_as_float((unsigned)(127 - 23 - (emax - e)) << 23));
  return __float2uint_ru(__fmul_ru(__fmul_ru(v, v), 268435456.0f));
}

// The RowStat of every (row, SCH k), part[c * R + r]: one read of x.  KFAST:
// one warp each, lanes along k; else a 32 x 8 block per 32 rows, lanes along
// rows.  (Two passes over the whole rows with atomics, the largest exponent
// first, read x twice: 0.8 of the 1.9 ms that 20 M elements took to convert.)
template <bool KFAST, bool K2>
__global__ void __launch_bounds__(256, 2) k_mod_stat(const ModView v, int64_t R, int64_t k, RowStat* __restrict__ part) {
  const int64_t nch = fricc_cdiv(k, (int64_t)SCH);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (KFAST) {
    for (int64_t w = (int64_t)blockIdx.x * 8 + warp; w < R * nch; w += (int64_t)gridDim.x * 8) {
      const int64_t r = w / nch, c = w - r * nch;
      const double* xr = v.x + v.rows.at(r);
      unsigned long long u[SCH / 32];
      int e = 0;
      unsigned cnt = 0, lo = ~0u;
#pragma unroll
      for (int q = 0; q < SCH / 32; ++q) {
        const int64_t j = c * SCH + 32 * q + lane;
        u[q] = j < k ? (unsigned long long)__double_as_longlong(__ldg(xr + koff<K2>(v, j))) : 0ull;
      }
#pragma unroll
      for (int q = 0; q < SCH / 32; ++q) {
        const int ej = exp_of(u[q]);
        e = ej > e ? ej : e;
        lo = min(lo, (unsigned)(ej - 1));
        cnt += ej ? 1u : 0u;
      }
      e = __reduce_max_sync(0xffffffffu, e);
      lo = __reduce_min_sync(0xffffffffu, lo);
      cnt = __reduce_add_sync(0xffffffffu, cnt);
      unsigned long long s = 0;
#pragma unroll
      for (int q = 0; q < SCH / 32; ++q) s += sq_units(u[q], e);
      s = warp_sum(s);
      if (lane == 0) part[c * R + r] = RowStat{s, e, (unsigned short)cnt, (unsigned short)lo};
    }
  } else {
    __shared__ unsigned long long ssum[8][33];
    __shared__ int se[8][33];
    __shared__ unsigned sc[8][33], sl[8][33];
    const int64_t nrb = fricc_cdiv(R, (int64_t)32);
    for (int64_t t = blockIdx.x; t < nrb * nch; t += gridDim.x) {
      const int64_t r = (t % nrb) * 32 + lane, c = t / nrb;
      unsigned long long u[SCH / 8];
      int e = 0;
      unsigned cnt = 0, lo = ~0u;
      const double* xr = v.x + (r < R ? v.rows.at(r) : 0);
#pragma unroll
      for (int q = 0; q < SCH / 8; ++q) {
        const int64_t j = c * SCH + 8 * q + warp;
        u[q] = r < R && j < k ? (unsigned long long)__double_as_longlong(__ldg(xr + koff<K2>(v, j))) : 0ull;
      }
#pragma unroll
      for (int q = 0; q < SCH / 8; ++q) {
        const int ej = exp_of(u[q]);
        e = ej > e ? ej : e;
        lo = min(lo, (unsigned)(ej - 1));
        cnt += ej ? 1u : 0u;
      }
      __syncthreads();
      se[warp][lane] = e;
      sc[warp][lane] = cnt;
      sl[warp][lane] = lo;
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 8; ++q) e = se[q][lane] > e ? se[q][lane] : e;
      unsigned long long s = 0;
#pragma unroll
      for (int q = 0; q < SCH / 8; ++q) s += sq_units(u[q], e);
      ssum[warp][lane] = s;
      __syncthreads();
      if (warp == 0 && r < R) {
        for (int q = 1; q < 8; ++q) {
          s += ssum[q][lane];
          cnt += sc[q][lane];
          lo = min(lo, sl[q][lane]);
        }
        part[c * R + r] = RowStat{s, e, (unsigned short)cnt, (unsigned short)lo};
      }
    }
  }
}

// the shift of each row: |x| 2^sh <= 2^61 for its norm (and > 2^60 but for
// subnormal rows)
__device__ __forceinline__ int shift_of(unsigned long long sum, int emax) {
  if (emax == 0) return 0;
  if (emax >= 2047) return SH_BAD;
  const int L = 64 - __clzll((long long)((sum - 1) | 1ull));  // sum <= 2^L
  return 61 - (emax - 1023 - 14 + (L + 1) / 2);
}

// A row's word of `cnt`: its nonzeros, and in the top byte how many binary places
// below the norm's bound 2^61 its smallest nonzero may lie (255: at least so
// many; a subnormal's own places count).
constexpr int SPAN_AT = 24;
__device__ __forceinline__ unsigned cnt_word(unsigned cnt, unsigned low, int sh) {
  if (cnt == 0 || sh == SH_BAD) return cnt;
  const int span = 61 - ((int)low - 1022 + sh) + (low == 0 ? 52 : 0);
  return cnt | (unsigned)min(max(span, 0), 255) << SPAN_AT;
}

// one warp per row: its parts combined (a long row has thousands)
__global__ void __launch_bounds__(256) k_mod_shift(const RowStat* __restrict__ part, int64_t R, int64_t nch,
                                                   int* __restrict__ sh, unsigned* __restrict__ cnt) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < R; r += (int64_t)gridDim.x * 8) {
    int e = 0;
    for (int64_t c = lane; c < nch; c += 32) {
      const int ec = part[c * R + r].emax;
      e = ec > e ? ec : e;
    }
    e = __reduce_max_sync(0xffffffffu, e);
    unsigned long long s = 0;
    unsigned n = 0, lo = ~0u;
    for (int64_t c = lane; c < nch; c += 32) {
      const RowStat p = part[c * R + r];
      if (p.cnt == 0) continue;
      lo = min(lo, (unsigned)p.low);
      const int d = 2 * (e - p.emax);
      s += d > 62 ? 1ull : (p.sum >> d) + 1ull;
      n += p.cnt;
    }
    s = warp_sum(s);
    n = __reduce_add_sync(0xffffffffu, n);
    lo = __reduce_min_sync(0xffffffffu, lo);
    if (lane == 0) {
      const int h = shift_of(s, e);
      sh[r] = h;
      cnt[r] = cnt_word(n, lo, h);
    }
  }
}

// X = rint(x 2^sh), |X| < 2^62
__device__ __forceinline__ long long scaled(double x, int sh) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int e = exp_of(u);
  if (e == 0 || sh == SH_BAD) return 0;
  const unsigned long long m = (u & 0xfffffffffffffull) | ((u >> 52) & 0x7ff ? 1ull << 52 : 0ull);
  const int s = e - 1075 + sh;  // <= 9
  unsigned long long v;
  if (s >= 0) v = m << s;
  else if (s > -56) v = ((m >> (-s - 1)) + 1) >> 1;  // half up
  else v = 0;
  return (long long)u < 0 ? -(long long)v : (long long)v;
}

// X0 and X1 in signed 16-bit digits (the leading one of 14 bits) as floats
__device__ __forceinline__ void digits(long long X0, long long X1, f32x2* d) {
  const unsigned long long b0 = (unsigned long long)X0 + 0x800080008000ull, b1 = (unsigned long long)X1 + 0x800080008000ull;
  const unsigned l0 = (unsigned)b0, l1 = (unsigned)b1, h0 = (unsigned)(b0 >> 32), h1 = (unsigned)(b1 >> 32);
  constexpr unsigned E = 0x4B00u;  // 2^23 + field
  const f32x2 bias = pk2(-8421376.0f, -8421376.0f);  // 2^23 + 2^15
  d[0] = add2(pk2(__uint_as_float(__byte_perm(l0, E, 0x5410)), __uint_as_float(__byte_perm(l1, E, 0x5410))), bias);
  d[1] = add2(pk2(__uint_as_float(__byte_perm(l0, E, 0x5432)), __uint_as_float(__byte_perm(l1, E, 0x5432))), bias);
  d[2] = add2(pk2(__uint_as_float(__byte_perm(h0, E, 0x5410)), __uint_as_float(__byte_perm(h1, E, 0x5410))), bias);
  d[3] = add2(pk2(__int_as_float(0x4B400000 + ((int)h0 >> 16)), __int_as_float(0x4B400000 + ((int)h1 >> 16))),
              pk2(-MAGIC, -MAGIC));
}

// The residues modulo the I-th modulus of SG pairs at once, two packed values an
// instruction, and the constants' registers set up once for all of them: three
// exact FMAs (sums below 2^15 (1 + 2 * 180) + 2^13 * 180 < 2^24) and one
// reduction.  One pair at a time with 13-bit digits and scalar FMAs, the
// conversion took 252 instructions an element and was bound by issuing them:
// 20 M elements 200 us, now 170.
constexpr int SG = 4;
template <int I>
__device__ __forceinline__ void put_residues(const f32x2 (*d)[4], const bool* live, __nv_bfloat16* at, int64_t step,
                                             int64_t plane) {
  if constexpr (I < NP) {
    constexpr float inv_ = 1.0f / (float)TAB.p[I], p_ = (float)TAB.p[I];
    constexpr float c0 = (float)TAB.c[I][0], c1 = (float)TAB.c[I][1], c2 = (float)TAB.c[I][2];
    const f32x2 inv = pk2(inv_, inv_), negp = pk2(-p_, -p_), k0 = pk2(c0, c0), k1 = pk2(c1, c1), k2 = pk2(c2, c2);
#pragma unroll
    for (int g = 0; g < SG; ++g) {
      const float2 r = upk2(reduce2(fma2(d[g][3], k2, fma2(d[g][2], k1, fma2(d[g][1], k0, d[g][0]))), inv, negp));
      if (live[g]) *reinterpret_cast<__nv_bfloat162*>(at + g * step) = __floats2bfloat162_rn(r.x, r.y);
    }
    put_residues<I + 1>(d, live, at + plane, step, plane);
  }
}

// Two adjacent k of each of SG rows (`step` elements apart) into every plane.
__device__ __forceinline__ void put_planes(const double (*x)[2], const int* sh, const bool* live, __nv_bfloat16* at,
                                           int64_t step, int64_t plane) {
  f32x2 d[SG][4];
#pragma unroll
  for (int g = 0; g < SG; ++g) digits(scaled(x[g][0], sh[g]), scaled(x[g][1], sh[g]), d[g]);
  // the squares of x 2^(sh - 61)
#pragma unroll
  for (int g = 0; g < SG; ++g) {
    f32x2 v = fma2(d[g][3], pk2(0x1p-13f, 0x1p-13f), mul2(d[g][2], pk2(0x1p-29f, 0x1p-29f)));
    v = fma2(d[g][1], pk2(0x1p-45f, 0x1p-45f), fma2(d[g][0], pk2(0x1p-61f, 0x1p-61f), v));
    const float2 q = upk2(mul2(v, v));
    if (live[g]) *reinterpret_cast<__nv_bfloat162*>(at + g * step + NP * plane) = __floats2bfloat162_rn(q.x, q.y);
  }
  put_residues<0>(d, live, at, step, plane);
}

// x -> its planes, in tiles of 32 rows x 64 k (4 KB of each plane); one warp
// writes a row of a tile.  KFAST: read along k; else the tile passes through
// shared memory.  Bound by the 32 bytes written per element.
template <bool KFAST, bool K2>
__global__ void __launch_bounds__(256, 3) k_mod_split(const ModView v, int64_t R, int64_t k, const int* __restrict__ sh,
                                                   __nv_bfloat16* __restrict__ planes) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nkb = fricc_cdiv(k, (int64_t)BK), nrb = fricc_cdiv(R, (int64_t)32);
  const int64_t plane = nkb * R * BK;
  __shared__ double t[KFAST ? 1 : 64][33];
  for (int64_t b = blockIdx.x; b < nrb * nkb; b += gridDim.x) {
    const int64_t kb = b / nrb, r0 = (b - kb * nrb) * 32, j0 = kb * BK;
    __nv_bfloat16* out = planes + (kb * R + r0) * BK + 2 * lane;
    double x[SG][2];
    int s[SG];
    bool live[SG];
    if (KFAST) {
      const int64_t j = j0 + 2 * lane;
#pragma unroll
      for (int q = 0; q < SG; ++q) {
        const int64_t r = r0 + warp + 8 * q;
        live[q] = r < R;
        const double* xr = v.x + (live[q] ? v.rows.at(r) : 0);
        x[q][0] = live[q] && j < k ? __ldg(xr + koff<K2>(v, j)) : 0.0;
        x[q][1] = live[q] && j + 1 < k ? __ldg(xr + koff<K2>(v, j + 1)) : 0.0;
        s[q] = live[q] ? sh[r] : 0;
      }
      put_planes(x, s, live, out + warp * BK, 8 * BK, plane);
    } else {
      __syncthreads();
      if (r0 + lane < R) {
        const double* xr = v.x + v.rows.at(r0 + lane);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int64_t j = j0 + warp + 8 * q;
          t[warp + 8 * q][lane] = j < k ? __ldg(xr + koff<K2>(v, j)) : 0.0;
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < SG; ++q) {
        const int rr = warp + 8 * q;
        live[q] = r0 + rr < R;
        x[q][0] = t[2 * lane][rr];
        x[q][1] = t[2 * lane + 1][rr];
        s[q] = live[q] ? sh[r0 + rr] : 0;
      }
      put_planes(x, s, live, out + warp * BK, 8 * BK, plane);
    }
  }
}

// The whole conversion of rows of at most SCH elements (t1's products, the
// O^2V^3 terms) in one read: 32 rows per block pass through shared memory,
// their statistics and shifts included.
template <bool KFAST, bool K2>
__global__ void __launch_bounds__(256, 3) k_mod_convert(const ModView v, int64_t R, int64_t k, int* __restrict__ sh,
                                                        unsigned* __restrict__ cnt,
                                                        __nv_bfloat16* __restrict__ planes) {
  extern __shared__ double ct[];  // [64 nkb][33]
  __shared__ unsigned long long ssum[8][33];
  __shared__ int se[8][33], ssh[32];
  __shared__ unsigned sc[8][33], sl[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nkb = (int)fricc_cdiv(k, (int64_t)BK), kp = nkb * BK, kk = (int)k;
  const int64_t nrb = fricc_cdiv(R, (int64_t)32), plane = nkb * R * BK;
  for (int64_t b = blockIdx.x; b < nrb; b += gridDim.x) {
    const int64_t r0 = b * 32;
    __syncthreads();
    if (KFAST) {
      for (int rr = warp; rr < 32; rr += 8) {
        const double* xr = v.x + (r0 + rr < R ? v.rows.at(r0 + rr) : 0);
        for (int j = lane; j < kp; j += 32)
          ct[j * 33 + rr] = r0 + rr < R && j < kk ? __ldg(xr + koff<K2>(v, j)) : 0.0;
      }
    } else {
      const double* xr = v.x + (r0 + lane < R ? v.rows.at(r0 + lane) : 0);
#pragma unroll 8
      for (int j = warp; j < kp; j += 8)
        ct[j * 33 + lane] = r0 + lane < R && j < kk ? __ldg(xr + koff<K2>(v, j)) : 0.0;
    }
    __syncthreads();
    int e = 0;
    unsigned n = 0, lo = ~0u;
    for (int j = warp; j < kk; j += 8) {
      const int ej = exp_of((unsigned long long)__double_as_longlong(ct[j * 33 + lane]));
      e = ej > e ? ej : e;
      lo = min(lo, (unsigned)(ej - 1));
      n += ej ? 1u : 0u;
    }
    se[warp][lane] = e;
    sc[warp][lane] = n;
    sl[warp][lane] = lo;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) e = se[q][lane] > e ? se[q][lane] : e;
    unsigned long long s = 0;
    for (int j = warp; j < kk; j += 8) s += sq_units((unsigned long long)__double_as_longlong(ct[j * 33 + lane]), e);
    ssum[warp][lane] = s;
    __syncthreads();
    if (warp == 0) {
      for (int q = 1; q < 8; ++q) {
        s += ssum[q][lane];
        n += sc[q][lane];
        lo = min(lo, sl[q][lane]);
      }
      const int h = shift_of(s, e);
      ssh[lane] = h;
      if (r0 + lane < R) {
        sh[r0 + lane] = h;
        cnt[r0 + lane] = cnt_word(n, lo, h);
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int kb = 0; kb < nkb; ++kb) {
      const int j = kb * BK + 2 * lane;
      double x[SG][2];
      int h[SG];
      bool live[SG];
#pragma unroll
      for (int q = 0; q < SG; ++q) {
        const int rr = warp + 8 * q;
        live[q] = r0 + rr < R;
        x[q][0] = ct[j * 33 + rr];
        x[q][1] = ct[(j + 1) * 33 + rr];
        h[q] = ssh[rr];
      }
      put_planes(x, h, live, planes + ((int64_t)kb * R + r0 + warp) * BK + 2 * lane, 8 * BK, plane);
    }
  }
}

// ------------------------------------------------------------ the GEMM
// n / d for n < 2^31 by a multiplication (host-made constants): every warp
// decodes every unit, and five integer divisions in each of 16 warps cost
// ~1000 issue slots a unit
struct FastDiv {
  unsigned mul = 0, shift = 0, d = 1;
  FastDiv() = default;
  explicit FastDiv(unsigned d_) : d(d_) {
    while ((1ull << shift) < d) ++shift;
    mul = (unsigned)(((1ull << 32) * ((1ull << shift) - d)) / d + 1);
  }
  __device__ __forceinline__ unsigned div(unsigned n) const { return (__umulhi(n, mul) + n) >> shift; }
};

struct GemmArgs {
  FastDiv by_rep, by_plane, by_slice, by_group, by_last;  // per_rep, per_plane, tiles, 16 tiles_n, tiles_m % 16
  int K, tiles_m, tiles_n, bn, stages;
  int a_box;             // rows of an A box: 128, or M rounded to 8 where that is less (the rest of the tile is not stored)
  int M;
  int a_rows, b_rows;    // rows of A and B (a K block of a plane)
  int a_rep, b_rep;      // rows per replica (0: shared)
  int ks, chunks;        // K slices, 512-wide K runs in all
  // the residues: [slice][plane][rep][ng][M][16], columns in groups of 16, so
  // that a warp's 32 rows store 1 KB runs (row-major, each lane's 16 bytes
  // went to a line of its own: 4096 store cycles a tile, the bound of every
  // product with a short K)
  int64_t ng, rep_stride, plane_stride, slice_stride;
  unsigned short* out;
};

struct Unit {
  int rep, plane, slice, mt, nt;
};
__device__ __forceinline__ Unit unit_of(const GemmArgs& g, int u) {
  Unit x;
  x.rep = (int)g.by_rep.div((unsigned)u);
  int w = u - x.rep * (int)g.by_rep.d;
  x.plane = (int)g.by_plane.div((unsigned)w);
  w -= x.plane * (int)g.by_plane.d;
  x.slice = (int)g.by_slice.div((unsigned)w);
  w -= x.slice * (int)g.by_slice.d;
  // tile_coords: groups of 16 M tiles sweep the N tiles
  const int gr = (int)g.by_group.div((unsigned)w), rem = w - gr * (int)g.by_group.d;
  const bool full = g.tiles_m - gr * 16 >= 16;
  x.nt = full ? rem >> 4 : (int)g.by_last.div((unsigned)rem);
  x.mt = gr * 16 + rem - x.nt * (full ? 16 : (int)g.by_last.d);
  return x;
}

// Work unit u = ((rep * PLANES + plane) * ks + slice) * tiles + tile.  Roles
// as in gemm_tc.cu: TMA producer, MMA issuer, sixteen epilogue warps; the two
// TMEM accumulators alternate per 512-wide K run, so a run is drained,
// reduced modulo p and added to the warps' registers while the next one
// accumulates.  A run of 128 x 256 outputs costs 4096 clocks of MMA and ~1700 of
// epilogue (plan_for).
__global__ void __launch_bounds__(MNT, 1)
    k_mod_gemm(const __grid_constant__ CUtensorMap tma, const __grid_constant__ CUtensorMap tmb, GemmArgs g, int nunits,
               unsigned* err) {
  extern __shared__ uint8_t dsm[];
  __shared__ __align__(8) uint64_t full[8], empty[8], tfull[2], tempty[2];
  __shared__ uint32_t tbase;
  __shared__ int failed;
  const int STAGES = g.stages;
  const uint32_t b_bytes = (uint32_t)g.bn * BK * 2, a_bytes = (uint32_t)g.a_box * BK * 2;
  const uint32_t base = (smem_u32(dsm) + 1023u) & ~1023u;
  const uint32_t sA = base, sB = base + STAGES * A_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = (g.K + BK - 1) / BK;
  const int cpk = (g.chunks + g.ks - 1) / g.ks;  // runs per slice

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&tfull[b]), 1);
      mbar_init(smem_u32(&tempty[b]), MEW);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tbase)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;

  if (warp == 0) {
    if (elect_one()) {  // TMA producer
      int q = 0, s = 0;  // k blocks issued over all units; stage q % STAGES
      uint32_t ph = 0;   // and its use's parity
      for (int u = blockIdx.x; u < nunits && !*(volatile int*)&failed; u += gridDim.x) {
        const Unit x = unit_of(g, u);
        const int ya = x.plane * nk * g.a_rows + x.rep * g.a_rep + x.mt * BM;
        const int yb = x.plane * nk * g.b_rows + x.rep * g.b_rep + x.nt * g.bn;
        const int kb1 = min(nk, (x.slice + 1) * cpk * KC);
        for (int kb = x.slice * cpk * KC; kb < kb1; ++kb, ++q) {
          if (q >= STAGES && !mbar_wait(smem_u32(&empty[s]), ph ^ 1u)) {
            atomicOr(err, FRICC_DEV_TIMEOUT);
            failed = 1;
            break;
          }
          mbar_expect_tx(smem_u32(&full[s]), a_bytes + b_bytes);
          tma_load_2d(sA + s * A_BYTES, &tma, 0, ya + kb * g.a_rows, smem_u32(&full[s]));
          tma_load_2d(sB + s * b_bytes, &tmb, 0, yb + kb * g.b_rows, smem_u32(&full[s]));
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      if (*(volatile int*)&failed) {
        // let the copies in flight land before the CTA's shared memory goes away
        for (int r = q - STAGES < 0 ? 0 : q - STAGES; r < q; ++r)
          mbar_wait(smem_u32(&full[r % STAGES]), (uint32_t)(r / STAGES) & 1u);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {  // MMA issuer
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(g.bn >> 3) << 17) |
                             ((uint32_t)(BM >> 4) << 24);
      // The chain wait, MMAs, commit of a k block must stay below its MMAs' time: no
      // division by the stage count, descriptors by one addition.  (With both and
      // a branch on the lane number it took ~900 clocks: 1204 TFLOP/s at 4500^3,
      // whatever the loads did; now ~400.)
      const uint64_t da = sw128_desc(sA), db = sw128_desc(sB);
      const uint32_t b_step = b_bytes >> 4;
      int i = 0, s = 0;  // runs; the stage
      uint32_t ph = 0;
      for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
        const int slice = unit_of(g, u).slice;
        const int kb1 = min(nk, (slice + 1) * cpk * KC);
        for (int kb0 = slice * cpk * KC; kb0 < kb1; kb0 += KC, ++i) {
          const int b = i & 1;
          // the epilogue must have drained this accumulator's previous run
          if (i >= 2 && !mbar_wait(smem_u32(&tempty[b]), ((uint32_t)(i >> 1) & 1u) ^ 1u)) {
            atomicOr(err, FRICC_DEV_TIMEOUT);
            failed = 1;
          }
          if (*(volatile int*)&failed) break;
          tc_fence_after();
          const uint32_t acc = tmem + (uint32_t)(b * 256);
          const int kb_end = min(kb1, kb0 + KC);
          for (int kb = kb0; kb < kb_end; ++kb) {
            if (!mbar_wait(smem_u32(&full[s]), ph)) {
              atomicOr(err, FRICC_DEV_TIMEOUT);
              failed = 1;
              break;
            }
            tc_fence_after();
            const uint64_t a0 = da + (uint32_t)s * (A_BYTES >> 4), b0 = db + (uint32_t)s * b_step;
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              tc_mma(acc, a0 + 2 * k, b0 + 2 * k, idesc, ((kb - kb0) | k) != 0);
            tc_commit(smem_u32(&empty[s]));
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
          tc_commit(smem_u32(&tfull[b]));  // arrives when this run's MMAs have completed
          if (*(volatile int*)&failed) break;
        }
        if (*(volatile int*)&failed) break;
      }
    }
  } else {  // epilogue warps: TMEM lanes 32 (warp % 4) ..., 16-column groups w4, w4 + 4, ...
    const int quad = warp & 3, w4 = (warp - 2) >> 2;
    int i = 0;
    bool stop = false;
    for (int u = blockIdx.x; u < nunits && !stop; u += gridDim.x) {
      const Unit x = unit_of(g, u);
      const bool sq = x.plane == NP;
      const float p = sq ? 1.0f : c_p[x.plane], iv = 1.0f / p;
      const f32x2 inv = pk2(iv, iv), negp = pk2(-p, -p);
      f32x2 acc[32];  // residues of the runs so far
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = 0ull;
      const int kb0 = x.slice * cpk * KC, kb1 = min(nk, kb0 + cpk * KC);
      for (int kb = kb0; kb < kb1; kb += KC, ++i) {
        const int b = i & 1;
        bool ok = mbar_wait(smem_u32(&tfull[b]), (uint32_t)(i >> 1) & 1u);
        ok = __all_sync(0xffffffffu, ok && !*(volatile int*)&failed);
        if (!ok) {
          if (lane == 0) {
            atomicOr(err, FRICC_DEV_TIMEOUT);
            failed = 1;
          }
          stop = true;
          break;
        }
        tc_fence_after();
        const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(b * 256 + w4 * 16);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if ((w4 + 4 * c) * 16 < g.bn) {
            float r[16];
            tc_ld16(at + (uint32_t)(c * 64), r);
            if (sq) {  // the largest run's sum
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float2 f = upk2(acc[c * 8 + j]);
                acc[c * 8 + j] = pk2(fmaxf(f.x, r[2 * j]), fmaxf(f.y, r[2 * j + 1]));
              }
            } else {  // (a run plus a residue stays below 2^24: 512 * 180^2 + 180)
#pragma unroll
              for (int j = 0; j < 8; ++j)
                acc[c * 8 + j] = reduce2(add2(acc[c * 8 + j], pk2(r[2 * j], r[2 * j + 1])), inv, negp);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&tempty[b]));
      }
      if (stop) break;
      const int64_t row = (int64_t)x.mt * BM + quad * 32 + lane;
      const int64_t cg = (int64_t)x.nt * (g.bn >> 4) + w4;
      unsigned short* o = g.out + x.slice * g.slice_stride + x.plane * g.plane_stride + x.rep * g.rep_stride +
                          (cg * g.M + row) * 16;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (row < g.M && (w4 + 4 * c) * 16 < g.bn && cg + 4 * c < g.ng) {
          uint32_t wd[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const f32x2 a = acc[c * 8 + j];
            if (sq) {
              const float2 f = upk2(a);
              const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
              wd[j] = *reinterpret_cast<const uint32_t*>(&h);
            } else {  // adding MAGIC leaves the integer in the low bits
              const float2 f = upk2(add2(a, pk2(MAGIC, MAGIC)));
              wd[j] = __byte_perm(__float_as_uint(f.x), __float_as_uint(f.y), 0x5410);
            }
          }
          uint4* d = reinterpret_cast<uint4*>(o + (int64_t)c * 64 * g.M);
          d[0] = make_uint4(wd[0], wd[1], wd[2], wd[3]);
          d[1] = make_uint4(wd[4], wd[5], wd[6], wd[7]);
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// ------------------------------------------------------------ the outputs
struct CombineArgs {
  const unsigned short* res;
  int64_t rep_stride, plane_stride;
  const int *sha, *shb;
  const unsigned *cnta, *cntb;
  int64_t a_rep, b_rep;
  int64_t M, N, K;
  ModOut out;
  int amode, bmode;     // alpha: 0 one, 1 minus one, 2 other; beta: 0 zero, 1 one, 2 other
  int col_fast;         // C is contiguous along its columns (else along its rows)
  const unsigned* err;  // the GEMM's error word: every tile to the list
  unsigned* count;      // the tiles with outputs to recompute,
  unsigned* list;       // and for each its number and a column mask per row
};
constexpr int LIST_W = 65;  // words of a list entry: the tile, 64 column bits per row

__device__ __forceinline__ void store_c(const CombineArgs& a, double* p, double x) {
  if (a.amode == 1) x = __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ull);
  else if (a.amode == 2) x = a.out.alpha * x;
  if (a.bmode == 0) *p = x;
  else if (a.bmode == 1) *p = x + *p;
  else *p = fma(a.out.beta, *p, x);
}

// v 2^e where that is subnormal or overflows (kept out of line: FP64
// instructions)
static __device__ __noinline__ double scaled_far(unsigned long long v, int e, bool neg) {
  const double x = scalbn((double)v, e);
  return neg ? -x : x;
}

// The Chinese remainder sum of 15 residues as a signed 96-bit fraction of M,
// times M 2^-sh, rounded once to FP64 (integers only: FP64 operations on
// this part cost more than the whole conversion).  *zero: the value is 0.
__device__ __forceinline__ double crt(const int* r, int sh, bool* zero) {
  long long a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    a0 += (long long)r[i] * TAB.f[i][0];
    a1 += (long long)r[i] * TAB.f[i][1];
    a2 += (long long)r[i] * TAB.f[i][2];
  }
  // limbs, lowest first, carries signed; bits above 96 wrap away
  const unsigned l0 = (unsigned)a0;
  a1 += a0 >> 32;
  const unsigned l1 = (unsigned)a1;
  const unsigned l2 = (unsigned)(a2 + (a1 >> 32));
  // |F| as three words, the top bits first
  const unsigned sg = (unsigned)((int)l2 >> 31);
  unsigned m0 = l0 ^ sg, m1 = l1 ^ sg, m2 = l2 ^ sg;
  if (sg) {
    m0 += 1u;
    m1 += m0 == 0u ? 1u : 0u;
    m2 += (m0 | m1) == 0u ? 1u : 0u;
  }
  int lz = 0;
  *zero = false;
  if (m2 == 0u) {  // a small value, or none: whole words first
    lz = 32;
    m2 = m1;
    m1 = m0;
    m0 = 0u;
    if (m2 == 0u) {
      lz = 64;
      m2 = m1;
      m1 = 0u;
      if (m2 == 0u) {
        *zero = true;
        return 0.0;
      }
    }
  }
  // the top 64 bits of the magnitude, normalised: |F| = t 2^(32 - lz)
  const int z = __clz((int)m2);
  lz += z;
  const unsigned long long t = ((unsigned long long)__funnelshift_l(m1, m2, z) << 32) | __funnelshift_l(m0, m1, z);
  unsigned long long v = __umul64hi(t, TAB.mtop);  // value = v 2^(62 - lz - sh)
  int be = 62 - lz - sh + 63 + 1023;
  if (!(v >> 63)) {
    v <<= 1;
    --be;
  }
  if (be < 1 || be > 2045) return scaled_far(v, be - 1086, sg != 0);
  const unsigned low = (unsigned)v & 0x7ffu;
  unsigned long long m = v >> 11;  // 53 bits
  m += (low + ((unsigned)m & 1u) > 0x400u) ? 1 : 0;  // half to even
  return __longlong_as_double((long long)((((unsigned long long)(be - 1) << 52) + m) | ((unsigned long long)sg << 63)));
}

// K slices: slice 0 = the sum of all (64 residues of at most 180), reduced to
// the residue one slice would have left, or of the squares the largest.  One grid
// row per plane; `words` of 2 values per plane, `slice` per slice.
__global__ void __launch_bounds__(256) k_mod_slices(unsigned* __restrict__ res, int64_t words, int64_t slice, int ks) {
  const int plane = blockIdx.y;
  res += plane * words;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < words; i += (int64_t)gridDim.x * 256) {
    const unsigned x = res[i];
    if (plane < NP) {
      int lo = (short)x, hi = (int)x >> 16;
#pragma unroll 8
      for (int s = 1; s < ks; ++s) {
        const unsigned y = res[i + s * slice];
        lo += (short)y;
        hi += (int)y >> 16;
      }
      const float p = c_p[plane], inv = 1.0f / p;
      lo -= (int)p * __float2int_rn((float)lo * inv);
      hi -= (int)p * __float2int_rn((float)hi * inv);
      res[i] = ((unsigned)lo & 0xffffu) | ((unsigned)hi << 16);
    } else {
      float lo = __uint_as_float(x << 16), hi = __uint_as_float(x & 0xffff0000u);
#pragma unroll 8
      for (int s = 1; s < ks; ++s) {
        const unsigned y = res[i + s * slice];
        lo = fmaxf(lo, __uint_as_float(y << 16));
        hi = fmaxf(hi, __uint_as_float(y & 0xffff0000u));
      }
      res[i] = (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xffff0000u);
    }
  }
}

constexpr float GUARD = 0x1p-16f;
// An output whose residues and whose sum of squares are zero is a true zero (no
// nonzero of its row meets one of its column) where one of the two is empty, or
// where the spans of both add up to no more than this: any two nonzeros that
// meet then leave a square of at least 2^-124 (2^-126 is the smallest normal FP32
// number).  Elsewhere the elements that meet may have been rounded to 0, or
// their squares may have underflowed beside integers that cancel.
constexpr unsigned ZERO_SPAN = 62;

// One 32 x 64 tile of outputs per step: residues in, C out, and an entry on
// the list for a tile with outputs to recompute (which are left alone).  A
// warp reads 256-byte runs: 8 rows of a 16-column group, four adjacent columns
// per lane (128-byte runs and two columns took 288 us for 900 x 22500 outputs, 264
// for 4500^2; now 231 and 244).  Its bytes (2 per plane in, 8-16 out per output)
// would take 140; ~290 instructions an output keep it from them.
// Masks: 64 column bits per row.
__device__ __forceinline__ bool masked(const unsigned char* row, int c) { return (row[c >> 3] >> (c & 7)) & 1u; }

__global__ void __launch_bounds__(256, 4) k_mod_combine(CombineArgs a, int64_t ntiles) {
  __shared__ double t[32][65];
  __shared__ __align__(4) unsigned char mask[32][8];
  __shared__ unsigned at;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tn = fricc_cdiv(a.N, (int64_t)64), per = fricc_cdiv(a.M, (int64_t)32) * tn;
  const bool gave_up = *a.err != 0;
  const int cg = warp & 3, cl = cg * 16 + 4 * (lane & 3);
  for (int64_t b = blockIdx.x; b < ntiles; b += gridDim.x) {
    const int64_t rep = b / per, w = b - rep * per;
    const int64_t r0 = (w / tn) * 32, c0 = (w % tn) * 64;
    const int64_t c = c0 + cl;
    int shb[4];
    unsigned nb[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      shb[h] = c + h < a.N ? a.shb[rep * a.b_rep + c + h] : 0;
      nb[h] = c + h < a.N ? a.cntb[rep * a.b_rep + c + h] : 0u;
    }
    unsigned any = 0;
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      const int rl = (warp >> 2) * 16 + 8 * q + (lane >> 2);
      const int64_t r = r0 + rl;
      unsigned no = 0;
      if (r < a.M && c < a.N) {  // (groups are whole: the other columns' residues exist)
        const unsigned short* res = a.res + rep * a.rep_stride + (((c0 >> 4) + cg) * a.M + r) * 16 + 4 * (lane & 3);
        uint2 w4[PLANES];
#pragma unroll
        for (int i = 0; i < PLANES; ++i) w4[i] = __ldg(reinterpret_cast<const uint2*>(res + i * a.plane_stride));
        const int sha = a.sha[rep * a.a_rep + r];
        const unsigned na = a.cnta[rep * a.a_rep + r];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          int ri[NP];
#pragma unroll
          for (int i = 0; i < NP; ++i) {
            const unsigned v = h < 2 ? w4[i].x : w4[i].y;
            ri[i] = h & 1 ? (int)v >> 16 : (int)(short)v;
          }
          const unsigned v = h < 2 ? w4[NP].x : w4[NP].y;
          const float s2 = __uint_as_float(h & 1 ? v & 0xffff0000u : v << 16);
          bool zero = false, bad = false;
          double x = 0.0;
          if (gave_up || sha == SH_BAD || shb[h] == SH_BAD) {
            bad = c + h < a.N;
          } else {
            x = crt(ri, sha + shb[h], &zero);
            const unsigned ka = na & ((1u << SPAN_AT) - 1), kb = nb[h] & ((1u << SPAN_AT) - 1);
            const float n = (float)(ka < kb ? ka : kb);
            bad = c + h < a.N && !(n * s2 >= GUARD);
            if (bad && zero && s2 == 0.0f) bad = n != 0.0f && (na >> SPAN_AT) + (nb[h] >> SPAN_AT) > ZERO_SPAN;
          }
          no |= bad ? 1u << h : 0u;
          t[rl][cl + h] = x;
        }
      }
      // the row's 16 bits of this group
      no <<= 4 * (lane & 3);
      no |= __shfl_xor_sync(0xffffffffu, no, 1);
      no |= __shfl_xor_sync(0xffffffffu, no, 2);
      if ((lane & 3) == 0) *reinterpret_cast<unsigned short*>(&mask[rl][2 * cg]) = (unsigned short)no;
      any |= no;
    }
    const bool bad = __syncthreads_or(any);
    if (bad) {
      if (threadIdx.x == 0) {
        at = atomicAdd(a.count, 1u) * LIST_W;
        a.list[at] = (unsigned)b;
      }
      __syncthreads();
      if (threadIdx.x < 64) a.list[at + 1 + threadIdx.x] = reinterpret_cast<const unsigned*>(mask)[threadIdx.x];
    }
    double* C = a.out.C + a.out.rep.at(rep);
    if (a.col_fast) {
      const bool in0 = c0 + lane < a.N, in1 = c0 + lane + 32 < a.N;
      const int64_t cc0 = in0 ? a.out.col.at(c0 + lane) : 0, cc1 = in1 ? a.out.col.at(c0 + lane + 32) : 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int rl = warp + 8 * q;
        if (r0 + rl >= a.M) break;
        double* row = C + a.out.row.at(r0 + rl);
        if (in0 && !(bad && masked(mask[rl], lane))) store_c(a, row + cc0, t[rl][lane]);
        if (in1 && !(bad && masked(mask[rl], lane + 32))) store_c(a, row + cc1, t[rl][lane + 32]);
      }
    } else if (r0 + lane < a.M) {
      const int64_t rr = a.out.row.at(r0 + lane);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int j = warp + 8 * q;
        if (c0 + j < a.N && !(bad && masked(mask[lane], j))) store_c(a, C + rr + a.out.col.at(c0 + j), t[lane][j]);
      }
    }
    __syncthreads();  // before the next tile's values and masks
  }
}

// The listed outputs with FP64 FMAs in k order (usually none: the kernel
// reads the count and returns).  With skip, elements of A (1) or B (2) whose
// bits are all zero are absent and multiply nothing.
__global__ void __launch_bounds__(256) k_mod_fix(CombineArgs a, const ModView A, const ModView B, int skip) {
  __shared__ double As[32][33], Bs[32][65];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t tn = fricc_cdiv(a.N, (int64_t)64), per = fricc_cdiv(a.M, (int64_t)32) * tn;
  const unsigned cnt = *a.count;
  for (unsigned l = blockIdx.x; l < cnt; l += gridDim.x) {
    const unsigned* entry = a.list + (int64_t)l * LIST_W;
    const int64_t b = entry[0], rep = b / per, w = b - rep * per;
    const int64_t r0 = (w / tn) * 32, c0 = (w % tn) * 64;
    double acc[2][4] = {};
    for (int64_t k0 = 0; k0 < a.K; k0 += 32) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // As[k][row], Bs[k][column]: lanes along the contiguous index
        const int ka = A.sk == 1 ? tx : ty + 8 * q, ma = A.sk == 1 ? ty + 8 * q : tx;
        As[ka][ma] = (r0 + ma < a.M && k0 + ka < a.K)
                         ? A.x[A.rows.at(rep * a.a_rep + r0 + ma) + A.kat(k0 + ka)] : 0.0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kb = B.sk == 1 ? tx : ty + 8 * q, nb = (B.sk == 1 ? ty + 8 * q : tx) + 32 * h;
          Bs[kb][nb] = (c0 + nb < a.N && k0 + kb < a.K)
                           ? B.x[B.rows.at(rep * a.b_rep + c0 + nb) + B.kat(k0 + kb)] : 0.0;
        }
      }
      __syncthreads();
      const int kn = a.K - k0 < 32 ? (int)(a.K - k0) : 32;
      for (int kk = 0; kk < kn; ++kk) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double y = Bs[kk][tx + 32 * h];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const double x = As[kk][ty + 8 * q];
            if (!skip || __double_as_longlong(skip == 1 ? x : y) != 0) acc[h][q] = fma(x, y, acc[h][q]);
          }
        }
      }
    }
    double* C = a.out.C + a.out.rep.at(rep);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int cl = tx + 32 * h;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int rl = ty + 8 * q;
        if (masked(reinterpret_cast<const unsigned char*>(entry + 1 + 2 * rl), cl))
          store_c(a, C + a.out.row.at(r0 + rl) + a.out.col.at(c0 + cl), acc[h][q]);
      }
    }
  }
}

// ------------------------------------------------------------ host
// The tile width and orientation by a model in clocks: rounds of units over
// the SMs times a unit's K steps or its drains, whichever is longer.  An MMA
// of 128 x bn x 16 takes bn/2 clocks of tensor pipe, ~100 of the issuing
// thread, and its operands 32 (128 + bn) bytes of L2 at the 68-74 per clock and
// SM that tiles of 96 to 256 columns were measured at (4500^3: 3.1 ms at 96, 2.3
// at 128, 1.77 at 224, 1.80 at 256); a drain issues ~6 clocks a column, ~1200
// clocks a unit overlap with nothing.  Pairs of CTAs on 256 x 256 tiles
// (cta_group::2: 49 bytes per clock) were 3% faster there and 5% slower at
// 400 x 10000 x 10000: the drains then set the pace.
struct Plan {
  int bn = 256, ks = 1;
  bool swap = false;
  double clocks = 0.0;
};
Plan plan_for(int64_t M, int64_t N, int64_t K, int64_t reps, int nsm) {
  Plan best;
  const int64_t nk = fricc_cdiv(K, BK), chunks = fricc_cdiv(nk, KC);
  for (int sw = 0; sw < 2; ++sw) {
    const int64_t m = sw ? N : M, n = sw ? M : N;
    for (int bn = 32; bn <= 256; bn += 16) {
      const int64_t tiles = fricc_cdiv(m, BM) * fricc_cdiv(n, bn) * PLANES * reps;
      int ks = 1;
      while (ks < MAX_KS && tiles * ks < 2 * nsm && chunks / (2 * ks) >= 2) ks *= 2;
      const double l2 = ((m < BM ? m : BM) + bn) * 32 / 70.0;
      double step = bn / 2 > 100 ? bn / 2 : 100;
      if (l2 > step) step = l2;
      const double runs = (double)fricc_cdiv(chunks, ks);
      const double mma = (nk < KC ? (double)nk : runs * KC) * 4.0 * step, drain = runs * (200.0 + 6.0 * bn);
      const double t = (double)fricc_cdiv(tiles * ks, nsm) * ((mma > drain ? mma : drain) + 1200.0);
      if (best.clocks == 0.0 || t < best.clocks) best = Plan{bn, ks, sw != 0, t};
    }
  }
  return best;
}

}  // namespace mod

int64_t fricc_mod_operand_bytes(int64_t rows, int64_t k) { return mod::layout(rows, k).bytes; }

template <bool KFAST, bool K2>
static int launch_operand(const ModView& v, int64_t rows, int64_t k, int* sh, unsigned* cnt, __nv_bfloat16* planes,
                          mod::RowStat* part, cudaStream_t st) {
  auto cap = [](int64_t n) { return (unsigned)(n < 152 * 16 ? (n < 1 ? 1 : n) : 152 * 16); };
  const int64_t nkb = fricc_cdiv(k, tc::BK), nrb = fricc_cdiv(rows, 32);
  if (k <= mod::SCH) {
    const int smem = (int)(nkb * tc::BK * 33 * sizeof(double));
    static std::atomic<bool> attr{false};
    if (!attr.load(std::memory_order_acquire)) {
      FRICC_CUDA(cudaFuncSetAttribute(mod::k_mod_convert<KFAST, K2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      mod::SCH * 33 * (int)sizeof(double)));
      attr.store(true, std::memory_order_release);
    }
    mod::k_mod_convert<KFAST, K2><<<cap(nrb), 256, smem, st>>>(v, rows, k, sh, cnt, planes);
    fricc_note_launch();
    return fricc_cuda_check(cudaGetLastError(), "mod operand");
  }
  const int64_t nch = fricc_cdiv(k, mod::SCH);
  mod::k_mod_stat<KFAST, K2><<<cap(KFAST ? fricc_cdiv(rows * nch, 8) : nrb * nch), 256, 0, st>>>(v, rows, k, part);
  mod::k_mod_shift<<<cap(fricc_cdiv(rows, 8)), 256, 0, st>>>(part, rows, nch, sh, cnt);
  mod::k_mod_split<KFAST, K2><<<cap(nrb * nkb), 256, 0, st>>>(v, rows, k, sh, planes);
  fricc_note_launch(3);
  return fricc_cuda_check(cudaGetLastError(), "mod operand");
}

// Scratch of a conversion (the statistics of rows of more than one part).
static int64_t part_bytes(int64_t rows, int64_t k) {
  return k <= mod::SCH ? 0 : rows * fricc_cdiv(k, mod::SCH) * (int64_t)sizeof(mod::RowStat);
}

static int convert(const ModView& v, int64_t rows, int64_t k, void* buf, void* part_buf, cudaStream_t st) {
  auto* part = static_cast<mod::RowStat*>(part_buf);
  const mod::Layout l = mod::layout(rows, k);
  int* sh = static_cast<int*>(buf);
  unsigned* cnt = reinterpret_cast<unsigned*>(static_cast<char*>(buf) + l.off_cnt);
  auto* planes = reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(buf) + l.off_planes);
  const bool kfast = v.sk == 1 || (v.rows.s0 != 1 && rows > 1);
  if (v.kn == 0)
    return kfast ? launch_operand<true, false>(v, rows, k, sh, cnt, planes, part, st)
                 : launch_operand<false, false>(v, rows, k, sh, cnt, planes, part, st);
  return kfast ? launch_operand<true, true>(v, rows, k, sh, cnt, planes, part, st)
               : launch_operand<false, true>(v, rows, k, sh, cnt, planes, part, st);
}

int fricc_mod_operand(const ModView& v, int64_t rows, int64_t k, void* buf, cudaStream_t st) {
  void* part = nullptr;
  const int64_t bytes = part_bytes(rows, k);
  int rc = bytes ? fricc_alloc(&part, bytes, st) : FRICC_OK;
  if (!rc) rc = convert(v, rows, k, buf, part, st);
  fricc_free(part, st);
  return rc;
}

double fricc_mod_time_us(int64_t M, int64_t N, int64_t K, int64_t reps, bool a_shared, bool b_shared, bool conv_a,
                         bool conv_b) {
  if (K < 1 || K > mod::MAX_K) return 1e30;
  // measured on a GB300: the product at the model's clocks (1.7 GHz) or at
  // 6 TB/s of planes, conversions at 10.5 ps an element, the combine at 12.5 ps
  // an output, ~8 us a kernel (its launch and scratch included: an o10v40
  // iteration is bound by the host)
  const mod::Plan p = mod::plan_for(M, N, K, reps, 152);
  const double kp = (double)fricc_cdiv(K, tc::BK) * tc::BK;
  const double ea = (double)(a_shared ? 1 : reps) * M * kp, eb = (double)(b_shared ? 1 : reps) * N * kp;
  const double planes = (ea + eb) * 2.0 * mod::PLANES / 6.0e6, mma = p.clocks / 1700.0;
  return (mma > planes ? mma : planes) + 10.5e-6 * ((conv_a ? ea : 0.0) + (conv_b ? eb : 0.0)) +
         12.5e-6 * (double)reps * M * N + 8.0 * (3 + (p.ks > 1) + ((conv_a ? 1 : 0) + (conv_b ? 1 : 0)) * (K > mod::SCH ? 3 : 1));
}

// The scratch of one product is bounded: where its planes and residues would
// take more than this, replicas are worked off in groups, and a single product
// in panels of the rows of its larger operand (the smaller one is converted
// whole).  All of it is taken before the first output is written, so a call that
// cannot have it is left to the caller's other kernel.
static constexpr int64_t MOD_PANEL_BYTES = 6ll << 30;
static thread_local int64_t g_scratch = -1;
int64_t fricc_mod_scratch_bound() { return g_scratch >= 0 ? g_scratch : MOD_PANEL_BYTES; }
extern "C" int fricc_mod_scratch(int64_t bytes) {
  if (bytes < -1) {
    fricc_set_error("mod_scratch: a number of bytes, 0 (no modular products) or -1 (the default bound)");
    return FRICC_ERR_ARG;
  }
  g_scratch = bytes;
  return FRICC_OK;
}

namespace {

// The buffers of a product's pieces, which follow each other on one stream:
// a first walk over the pieces finds the largest of each.
struct Scratch {
  enum { WHOLE, OPA, OPB, PART, RES, WORDS, N };
  bool sizing = true;
  int64_t need[N] = {};
  void* buf[N] = {};
  // the last piece's plan, which the second walk mostly asks for again (~3 us)
  int64_t shape[4] = {};
  mod::Plan plan;
  const mod::Plan& plan_of(int64_t M, int64_t Nn, int64_t K, int64_t reps, int nsm) {
    if (shape[0] != M || shape[1] != Nn || shape[2] != K || shape[3] != reps) {
      plan = mod::plan_for(M, Nn, K, reps, nsm);
      shape[0] = M;
      shape[1] = Nn;
      shape[2] = K;
      shape[3] = reps;
    }
    return plan;
  }
  void* take(int which, int64_t bytes) {
    if (sizing && bytes > need[which]) need[which] = bytes;
    return buf[which];
  }
  int get(cudaStream_t st) {
    sizing = false;
    for (int k = 0; k < N; ++k)
      if (need[k])
        if (int rc = fricc_alloc(&buf[k], need[k], st)) return rc;
    return FRICC_OK;
  }
  void give_back(cudaStream_t st) {
    for (int k = 0; k < N; ++k) fricc_free(buf[k], st);
  }
};

// One launch of each kernel.  (sizing: only the scratch it takes; FRICC_MOD_NONE
// where it is too large for one launch.)
int mod_piece(const ModView& A, const ModView& B, const ModOut& out_, int64_t M, int64_t N, int64_t K, int64_t reps,
              bool a_shared, bool b_shared, bool skip_zero, Scratch& scr, cudaStream_t st) {
  const int64_t rows_a = (a_shared ? 1 : reps) * M, rows_b = (b_shared ? 1 : reps) * N;
  const mod::Layout la = mod::layout(rows_a, K), lb = mod::layout(rows_b, K);
  int nsm = 0;
  int rc = tc::sm_count(&nsm);
  if (rc) return rc;
  const mod::Plan pl = scr.plan_of(M, N, K, reps, nsm);
  const bool sw = pl.swap;  // the residues as [N][M] instead of [M][N]
  const int64_t m = sw ? N : M, n = sw ? M : N;
  const int64_t tm = fricc_cdiv(m, tc::BM), tn = fricc_cdiv(n, pl.bn);
  const int64_t nk = fricc_cdiv(K, tc::BK), chunks = fricc_cdiv(nk, mod::KC);
  const int a_box = (int)(m < tc::BM ? fricc_cdiv(m, 8) * 8 : tc::BM);
  const int ks = (int)fricc_cdiv(chunks, fricc_cdiv(chunks, pl.ks));  // every slice non-empty
  const int64_t ng = fricc_cdiv(n, 16);
  const int64_t units = tm * tn * mod::PLANES * reps * ks;
  const int64_t tiles = reps * fricc_cdiv(m, 32) * fricc_cdiv(n, 64);
  if (units > 0x7fffffff || tiles * mod::LIST_W > 0x7fffffff || mod::PLANES * nk * rows_a + 256 > 0x7fffffff ||
      mod::PLANES * nk * rows_b + 256 > 0x7fffffff)
    return FRICC_MOD_NONE;
  void* bufa = A.prepared ? nullptr : scr.take(Scratch::OPA, la.bytes);
  void* bufb = B.prepared ? nullptr : scr.take(Scratch::OPB, lb.bytes);
  void* part = scr.take(Scratch::PART, A.prepared ? 0 : part_bytes(rows_a, K));
  part = scr.take(Scratch::PART, B.prepared ? 0 : part_bytes(rows_b, K));
  auto* res = static_cast<unsigned short*>(
      scr.take(Scratch::RES, (int64_t)ks * mod::PLANES * reps * m * ng * 16 * (int64_t)sizeof(unsigned short)));
  // error word, list length, list
  auto* words = static_cast<unsigned*>(scr.take(Scratch::WORDS, (2 + tiles * mod::LIST_W) * (int64_t)sizeof(unsigned)));
  if (scr.sizing) return FRICC_OK;
  if (!A.prepared) rc = convert(A, rows_a, K, bufa, part, st);
  if (!rc && !B.prepared) rc = convert(B, rows_b, K, bufb, part, st);
  if (!rc) rc = fricc_cuda_check(cudaMemsetAsync(words, 0, 2 * sizeof(unsigned), st), "mod_gemm");
  if (!rc) {
    const char* pa = static_cast<const char*>(A.prepared ? A.prepared : bufa);
    const char* pb = static_cast<const char*>(B.prepared ? B.prepared : bufb);
    const int64_t ra = a_shared ? 0 : M, rb = b_shared ? 0 : N;
    CUtensorMap ma, mb;
    const char *qa = sw ? pb : pa, *qb = sw ? pa : pb;
    const mod::Layout &xa = sw ? lb : la, &xb = sw ? la : lb;
    rc = tc::make_map(&ma, qa + xa.off_planes, mod::PLANES * xa.nkb * xa.rows, tc::BK, tc::BK, a_box);
    if (!rc) rc = tc::make_map(&mb, qb + xb.off_planes, mod::PLANES * xb.nkb * xb.rows, tc::BK, tc::BK, pl.bn);
    if (!rc) {
      constexpr int SMEM = 226 * 1024;  // + 0.2 KB of barriers
      mod::GemmArgs g{};
      g.K = (int)K;
      g.tiles_m = (int)tm;
      g.tiles_n = (int)tn;
      g.bn = pl.bn;
      g.a_box = a_box;
      const int stage = tc::A_BYTES + pl.bn * tc::BK * 2;
      g.stages = (SMEM - 1024) / stage < 8 ? (SMEM - 1024) / stage : 8;
      g.M = (int)m;
      g.a_rows = (int)xa.rows;
      g.b_rows = (int)xb.rows;
      g.a_rep = (int)(sw ? rb : ra);
      g.b_rep = (int)(sw ? ra : rb);
      g.ks = ks;
      g.chunks = (int)chunks;
      g.by_rep = mod::FastDiv((unsigned)(tm * tn * ks * mod::PLANES));
      g.by_plane = mod::FastDiv((unsigned)(tm * tn * ks));
      g.by_slice = mod::FastDiv((unsigned)(tm * tn));
      g.by_group = mod::FastDiv((unsigned)(16 * tn));
      g.by_last = mod::FastDiv((unsigned)(tm % 16 ? tm % 16 : 16));
      g.ng = ng;
      g.rep_stride = m * ng * 16;
      g.plane_stride = reps * g.rep_stride;
      g.slice_stride = mod::PLANES * g.plane_stride;
      g.out = res;
      static std::atomic<bool> attr{false};
      cudaError_t e = cudaSuccess;
      if (!attr.load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(mod::k_mod_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e == cudaSuccess) attr.store(true, std::memory_order_release);
      }
      if (e == cudaSuccess) {
        const bool prof = fricc_prof_on();
        if (prof) fricc_prof_record(st, true, 0.0, 1);
        const unsigned grid = (unsigned)(units < nsm ? units : nsm);
        mod::k_mod_gemm<<<grid, mod::MNT, g.stages * stage + 1024, st>>>(ma, mb, g, (int)units, words);
        if (prof) fricc_prof_record(st, false, 2.0 * mod::PLANES * (double)reps * (double)M * (double)N * (double)K, 1);
        mod::CombineArgs c{};
        c.res = res;
        c.rep_stride = g.rep_stride;
        c.plane_stride = g.plane_stride;
        c.sha = reinterpret_cast<const int*>(qa);
        c.shb = reinterpret_cast<const int*>(qb);
        c.cnta = reinterpret_cast<const unsigned*>(qa + xa.off_cnt);
        c.cntb = reinterpret_cast<const unsigned*>(qb + xb.off_cnt);
        c.a_rep = g.a_rep;
        c.b_rep = g.b_rep;
        c.M = m;
        c.N = n;
        c.K = K;
        c.out = out_;
        if (sw) {
          c.out.row = out_.col;
          c.out.col = out_.row;
        }
        c.amode = out_.alpha == 1.0 ? 0 : (out_.alpha == -1.0 ? 1 : 2);
        c.bmode = out_.beta == 0.0 ? 0 : (out_.beta == 1.0 ? 1 : 2);
        c.col_fast = c.out.col.s0 == 1 || c.out.row.s0 != 1;
        c.err = words;
        c.count = words + 1;
        c.list = words + 2;
        if (ks > 1) {
          const int64_t gs = fricc_cdiv(g.plane_stride / 2, 256);
          mod::k_mod_slices<<<dim3((unsigned)(gs < 152 ? gs : 152), mod::PLANES), 256, 0, st>>>(
              reinterpret_cast<unsigned*>(res), g.plane_stride / 2, g.slice_stride / 2, ks);
          fricc_note_launch();
        }
        const unsigned gc = (unsigned)(tiles < 152 * 8 ? tiles : 152 * 8);
        mod::k_mod_combine<<<gc, 256, 0, st>>>(c, tiles);
        // the recomputation reads the operands in the orientation of the residues;
        // "absent" elements are those of the caller's A
        const ModView &fa = sw ? B : A, &fb = sw ? A : B;
        mod::k_mod_fix<<<152 * 4, 256, 0, st>>>(c, fa, fb, skip_zero ? (sw ? 2 : 1) : 0);
        fricc_note_launch(3);
        e = cudaGetLastError();
      }
      if (e != cudaSuccess) rc = fricc_cuda_fail(e, "mod_gemm", __FILE__, __LINE__);
    }
  }
  return rc;
}

// A single product, in panels where it has to be.
int mod_single(const ModView& A, const ModView& B, const ModOut& out, int64_t M, int64_t N, int64_t K, bool skip_zero,
               Scratch& scr, cudaStream_t st) {
  // (a prepared operand's planes are not cut: the other one's rows are)
  const int64_t bound = fricc_mod_scratch_bound(), least = g_scratch >= 0 ? 256 : 1024;
  const bool cut_b = !B.prepared && (A.prepared || N >= M);
  const int64_t len = cut_b ? N : M;
  const int64_t per_row = 2 * mod::PLANES * ((cut_b ? M : N) + fricc_cdiv(K, 64) * 64);
  if ((cut_b ? B : A).prepared || len <= 2 * least || len * per_row <= bound)
    return mod_piece(A, B, out, M, N, K, 1, true, true, skip_zero, scr, st);
  int64_t panel = bound / per_row / 256 * 256;
  if (panel < least) panel = least;
  ModView whole = cut_b ? A : B;
  int rc = FRICC_OK;
  if (!whole.prepared) {
    const int64_t rows = cut_b ? M : N;
    void* buf = scr.take(Scratch::WHOLE, fricc_mod_operand_bytes(rows, K));
    void* part = scr.take(Scratch::PART, part_bytes(rows, K));
    if (!scr.sizing) rc = convert(whole, rows, K, buf, part, st);
    whole.prepared = scr.sizing ? static_cast<const void*>(&scr) : buf;  // (not read while sizing)
  }
  for (int64_t r0 = 0; r0 < len && !rc; r0 += panel) {
    const int64_t n = len - r0 < panel ? len - r0 : panel;
    ModView cut = cut_b ? B : A;
    ModOut o = out;
    cut.rows.off += r0;
    (cut_b ? o.col : o.row).off += r0;
    rc = cut_b ? mod_piece(whole, cut, o, M, n, K, 1, true, true, skip_zero, scr, st)
               : mod_piece(cut, whole, o, n, N, K, 1, true, true, skip_zero, scr, st);
  }
  return rc;
}

// The replicas, in groups where they have to be.
int mod_groups(const ModView& A, const ModView& B, const ModOut& out, int64_t M, int64_t N, int64_t K, int64_t reps,
               bool a_shared, bool b_shared, bool skip_zero, Scratch& scr, cudaStream_t st) {
  if (reps == 1) return mod_single(A, B, out, M, N, K, skip_zero, scr, st);
  const int64_t kp = fricc_cdiv(K, 64) * 64;
  const int64_t per = 2 * mod::PLANES * (M * N + (a_shared ? 0 : M * kp) + (b_shared ? 0 : N * kp));
  int64_t group = fricc_mod_scratch_bound() / per;
  if (group >= reps) return mod_piece(A, B, out, M, N, K, reps, a_shared, b_shared, skip_zero, scr, st);
  if (group < 1) group = 1;
  int rc = FRICC_OK;
  for (int64_t r0 = 0; r0 < reps && !rc; r0 += group) {
    const int64_t n = reps - r0 < group ? reps - r0 : group;
    ModView a = A, b = B;
    ModOut o = out;
    if (!a_shared) a.rows.off += r0 * M;
    if (!b_shared) b.rows.off += r0 * N;
    o.rep.off += r0;
    rc = n == 1 ? mod_single(a, b, o, M, N, K, skip_zero, scr, st)
                : mod_piece(a, b, o, M, N, K, n, a_shared, b_shared, skip_zero, scr, st);
  }
  return rc;
}

}  // namespace

int fricc_mod_gemm(const ModView& A, const ModView& B, const ModOut& out, int64_t M, int64_t N, int64_t K, int64_t reps,
                   bool a_shared, bool b_shared, bool skip_zero, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0 || K > mod::MAX_K || reps < 1) {
    fricc_set_error("mod_gemm: bad arguments");
    return FRICC_ERR_ARG;
  }
  if (fricc_mod_scratch_bound() == 0) return FRICC_MOD_NONE;
  Scratch scr;
  int rc = mod_groups(A, B, out, M, N, K, reps, a_shared, b_shared, skip_zero, scr, st);
  if (rc) return rc;
  rc = scr.get(st) ? FRICC_MOD_NONE : mod_groups(A, B, out, M, N, K, reps, a_shared, b_shared, skip_zero, scr, st);
  scr.give_back(st);
  return rc;
}

// The FP64 tiles run at ~1.0 TFLOP/s on their padded shape (0.73-0.92 of the
// FP64 rate over the iteration's shapes), the FP32-pair ones at ~2.5; ~10 us
// at least.
double fricc_mod_alt_us(int64_t batch, int64_t M, int64_t N, int64_t K, bool pairs) {
  const double pad = (double)(fricc_cdiv(M, 32) * 32) * (double)(fricc_cdiv(N, 32) * 32);
  return 10.0 + 2.0 * (double)batch * pad * (double)K / (pairs ? 2.5e6 : 1.0e6);
}

bool fricc_mod_chosen(int64_t batch, int64_t M, int64_t N, int64_t K, bool a_batched, bool b_batched, bool a_prepared,
                      bool b_prepared, double alt_us) {
  const int force = fricc_mod_mode();
  // (up to four rows or columns are the GEMV kernels'; a tile set by a tuner is a
  // choice of the other kernels)
  if (force == 0 || M <= 4 || N <= 4 || K > mod::MAX_K || fricc_tune_get(FRICC_TUNE_GEMM_TILE) >= 0) return false;
  if (force == 1) return true;
  int64_t reps = 1;
  if (batch > 1) {
    if (a_batched && b_batched) reps = batch;
    else if (b_batched) N *= batch;
    else M *= batch;
  }
  return fricc_mod_time_us(M, N, K, reps, reps == 1, reps == 1, !a_prepared, !b_prepared) < 0.8 * alt_us;
}

int fricc_mod_try(const double* A, const double* B, double* C, int64_t batch, int64_t batch2, int64_t M, int64_t N,
                  int64_t K, const int64_t sA[3], const int64_t sB[3], const int64_t sC[3], const int64_t* s2,
                  double alpha, double beta, bool pairs, const void* a_mod, const void* b_mod, cudaStream_t st) {
  if (!fricc_mod_chosen(batch, M, N, K, sA[2] != 0, sB[2] != 0, a_mod != nullptr, b_mod != nullptr,
                        fricc_mod_alt_us(batch, M, N, K, pairs)))
    return FRICC_MOD_NONE;
  struct Level {
    int64_t n, a, b, c;
  };
  const Level lv[2] = {{batch, sA[2], sB[2], sC[2]}, {batch2, s2 ? s2[0] : 0, s2 ? s2[1] : 0, s2 ? s2[2] : 0}};
  ModView va, vb;
  ModOut out;
  va.x = A;
  va.sk = sA[1];
  va.rows.outer(M, sA[0]);
  va.prepared = a_mod;
  vb.x = B;
  vb.sk = sB[0];
  vb.rows.outer(N, sB[1]);
  vb.prepared = b_mod;
  out.C = C;
  out.alpha = alpha;
  out.beta = beta;
  out.row.outer(M, sC[0]);
  out.col.outer(N, sC[1]);
  int64_t m = M, n = N, reps = 1;
  // a level that moves only A (or only B) is flattened into its rows; the
  // levels that move both follow: replicas are the slowest index of the rows.
  // One that moves neither repeats A's rows, or, where those are prepared, B's:
  // a prepared operand has its own rows and no more.
  for (int k = 0; k < 2; ++k) {
    const Level& l = lv[k];
    if (l.n == 1 || (l.a != 0 && l.b != 0)) continue;
    if (l.a == 0 && l.b == 0 && a_mod) vb.prepared = nullptr;
    if (l.b == 0 && !(l.a == 0 && a_mod)) {
      va.rows.outer(l.n, l.a);
      out.row.outer(l.n, l.c);
      m *= l.n;
    } else {
      vb.rows.outer(l.n, l.b);
      out.col.outer(l.n, l.c);
      n *= l.n;
    }
  }
  for (const Level& l : lv) {
    if (l.n == 1 || l.a == 0 || l.b == 0) continue;
    va.rows.outer(l.n, l.a);
    vb.rows.outer(l.n, l.b);
    out.rep.outer(l.n, l.c);
    reps *= l.n;
  }
  return fricc_mod_gemm(va, vb, out, m, n, K, reps, reps == 1, reps == 1, false, st);
}
