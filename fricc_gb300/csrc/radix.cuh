// Stable sorts of (uint64 key, uint32 value) pairs on the FRI path: an LSD
// radix sort, 8-bit digits, that buckets the nonzeros of a SparseTensor4d by an
// index pair while keeping nonzero-slot order inside each bucket (the
// accumulation order of src/sparse_tensor.cpp), and below it the descending sort
// of a compression's candidates by |x| with ties in ascending flat index (the
// order a stable merge sort by |x| gives, fri-cc src/fri_utils.cpp:22-25).
#pragma once
#include "common.cuh"

namespace radix {

constexpr int NT = 256;
constexpr int IPT = 8;
constexpr int TILE = NT * IPT;

__device__ __forceinline__ unsigned digit(unsigned long long k, int shift) { return (unsigned)(k >> shift) & 255u; }

// Replica batches: blockIdx.y (blockIdx.x for k_scan_digits) is the replica;
// its keys and values start kv_stride elements after the previous one's,
// its histogram hist_stride words after, its element count (of the sort that
// reads it from the device) n_stride int64s after.
struct Batch {
  int64_t kv_stride = 0, hist_stride = 0, n_stride = 0;
};

static __global__ void __launch_bounds__(NT) k_hist(const unsigned long long* __restrict__ keys, int64_t n, int shift,
                                             unsigned* __restrict__ hist, int64_t ntiles, Batch bt) {
  const int rep = blockIdx.y;
  keys += rep * bt.kv_stride;
  hist += rep * bt.hist_stride;
  __shared__ unsigned h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * TILE;
#pragma unroll
  for (int r = 0; r < IPT; ++r) {
    const int64_t i = base + r * NT + threadIdx.x;
    if (i < n) atomicAdd(&h[digit(keys[i], shift)], 1u);
  }
  __syncthreads();
  hist[(int64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of each digit's per-tile counts (one block per digit, in
// place); the digit's total goes to totals[d].
static __global__ void __launch_bounds__(256) k_scan_rows(unsigned* hist, int64_t ntiles, unsigned* totals, Batch bt) {
  hist += blockIdx.y * bt.hist_stride;
  totals += blockIdx.y * bt.hist_stride;
  __shared__ int64_t sm[33];
  unsigned* row = hist + (int64_t)blockIdx.x * ntiles;
  const int64_t per = fricc_cdiv(ntiles, 256);
  const int64_t b = threadIdx.x * per;
  const int64_t e = b + per < ntiles ? b + per : ntiles;
  int64_t loc = 0;
  for (int64_t i = b; i < e; ++i) loc += row[i];
  int64_t tot;
  int64_t run = block_excl_sum(loc, sm, &tot);
  for (int64_t i = b; i < e; ++i) {
    const unsigned c = row[i];
    row[i] = (unsigned)run;
    run += c;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = (unsigned)tot;
}

// Exclusive scan of the 256 digit totals into base[d].
static __global__ void __launch_bounds__(256) k_scan_digits(const unsigned* totals, unsigned* base, Batch bt) {
  totals += blockIdx.x * bt.hist_stride;
  base += blockIdx.x * bt.hist_stride;
  __shared__ int64_t sm[33];
  int64_t tot;
  base[threadIdx.x] = (unsigned)block_excl_sum(totals[threadIdx.x], sm, &tot);
}

static __global__ void __launch_bounds__(NT) k_scatter(const unsigned long long* __restrict__ kin,
                                                const unsigned* __restrict__ vin,
                                                unsigned long long* __restrict__ kout, unsigned* __restrict__ vout,
                                                int64_t n, int shift, const unsigned* __restrict__ offs, int64_t ntiles,
                                                const unsigned* __restrict__ dbase, Batch bt) {
  const int rep = blockIdx.y;
  kin += rep * bt.kv_stride;
  vin += rep * bt.kv_stride;
  kout += rep * bt.kv_stride;
  vout += rep * bt.kv_stride;
  offs += rep * bt.hist_stride;
  dbase += rep * bt.hist_stride;
  constexpr int NW = NT / 32;
  __shared__ unsigned run[256];
  __shared__ unsigned wc[NW][256];
  run[threadIdx.x] = dbase[threadIdx.x] + offs[(int64_t)threadIdx.x * ntiles + blockIdx.x];
  unsigned lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  const int w = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * TILE;
  for (int r = 0; r < IPT; ++r) {
#pragma unroll
    for (int k = 0; k < NW; ++k) wc[k][threadIdx.x] = 0;
    __syncthreads();
    const int64_t i = base + r * NT + threadIdx.x;
    const bool valid = i < n;
    unsigned long long key = 0;
    unsigned val = 0;
    unsigned d = 256;
    if (valid) {
      key = kin[i];
      val = vin[i];
      d = digit(key, shift);
    }
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const unsigned lrank = __popc(peers & lt);
    if (valid && lrank == 0) wc[w][d] = __popc(peers);
    __syncthreads();
    {
      unsigned acc = run[threadIdx.x];
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const unsigned c = wc[k][threadIdx.x];
        wc[k][threadIdx.x] = acc;
        acc += c;
      }
      run[threadIdx.x] = acc;
    }
    __syncthreads();
    if (valid) {
      const unsigned pos = wc[w][d] + lrank;
      kout[pos] = key;
      vout[pos] = val;
    }
    __syncthreads();
  }
}

// Sorts n pairs on key bits [0, bits), ascending.
// The result ends in (keys, vals); the tmp buffers must hold n entries, hist
// hist_words(n) counts.
inline int64_t hist_words(int64_t n) { return 256 * fricc_cdiv(n, TILE) + 512; }

// With R > 1, R independent sorts of the replicas' arrays (kv_stride apart,
// each n long; hist holds R * hist_stride words, hist_stride >=
// hist_words(n)).
inline int sort_pairs(unsigned long long* keys, unsigned* vals, unsigned long long* ktmp, unsigned* vtmp,
                      int64_t n, int bits, unsigned* hist, cudaStream_t st, int R = 1, Batch bt = Batch{}) {
  if (n <= 1) return FRICC_OK;
  if (n > 0xffffffffLL || R < 1 || R > 65535) return FRICC_ERR_ARG;
  const int64_t ntiles = fricc_cdiv(n, TILE);
  unsigned long long *ka = keys, *kb = ktmp;
  unsigned *va = vals, *vb = vtmp;
  int passes = 0;
  for (int shift = 0; shift < bits; shift += 8, ++passes) {
    unsigned* totals = hist + 256 * ntiles;
    unsigned* base = totals + 256;
    k_hist<<<dim3((unsigned)ntiles, (unsigned)R), NT, 0, st>>>(ka, n, shift, hist, ntiles, bt);
    k_scan_rows<<<dim3(256, (unsigned)R), 256, 0, st>>>(hist, ntiles, totals, bt);
    k_scan_digits<<<R, 256, 0, st>>>(totals, base, bt);
    k_scatter<<<dim3((unsigned)ntiles, (unsigned)R), NT, 0, st>>>(ka, va, kb, vb, n, shift, hist, ntiles, base,
                                                                  bt);
    fricc_note_launch(4);
    unsigned long long* tk = ka;
    ka = kb;
    kb = tk;
    unsigned* tv = va;
    va = vb;
    vb = tv;
  }
  FRICC_LAUNCH_CHECK();
  if (passes & 1) {
    const int64_t span = R > 1 ? (int64_t)(R - 1) * bt.kv_stride + n : n;
    FRICC_CUDA(cudaMemcpyAsync(keys, ka, span * sizeof(unsigned long long), cudaMemcpyDeviceToDevice, st));
    FRICC_CUDA(cudaMemcpyAsync(vals, va, span * sizeof(unsigned), cudaMemcpyDeviceToDevice, st));
  }
  return FRICC_OK;
}

// ---------------------------------------------------------------------------
// The descending sort of a compression's candidates, whose count only the
// device knows, in two launches instead of 32 (8 digits x 4 kernels, of
// which a small sort is all launch latency: 185 us for 20,000 keys).
//
// Up to RANK_MAX candidates (D of an MP2-like tensor is a few thousand
// entries): each element's place is the number of elements before it,
// counted directly, n^2 comparisons spread over the chip (36 us at 16384,
// 3 us at 2000).  Above that the digits pass in one cooperative kernel
// with a barrier between the steps of a pass.  The kernel that has nothing
// to do returns at once.
constexpr int64_t RANK_MAX = 16384;
constexpr int RANK_I = 64;  // elements placed by one block of 256: 4 threads share one

// dst = src sorted by descending key, equal keys in source order
static __global__ void __launch_bounds__(256) k_rank_sort(const unsigned long long* __restrict__ ksrc,
                                                          const unsigned* __restrict__ vsrc,
                                                          unsigned long long* __restrict__ kdst,
                                                          unsigned* __restrict__ vdst,
                                                          const int64_t* __restrict__ n_dev, Batch bt) {
  const int rep = blockIdx.y;
  const int64_t n = n_dev[rep * bt.n_stride];
  const int64_t i0 = (int64_t)blockIdx.x * RANK_I;
  if (n > RANK_MAX || i0 >= n) return;
  ksrc += rep * bt.kv_stride;
  vsrc += rep * bt.kv_stride;
  kdst += rep * bt.kv_stride;
  vdst += rep * bt.kv_stride;
  constexpr int T = 1024;
  __shared__ unsigned long long sk[T];
  __shared__ int part[4][RANK_I];
  const int ii = threadIdx.x & (RANK_I - 1), q = threadIdx.x / RANK_I;  // a warp shares q: sk reads broadcast
  const int i = (int)i0 + ii;
  const unsigned long long ki = i < n ? ksrc[i] : 0ull;
  int before = 0;
  for (int t0 = 0; t0 < n; t0 += T) {
    __syncthreads();
    for (int j = threadIdx.x; j < T; j += 256) sk[j] = t0 + j < n ? ksrc[t0 + j] : 0ull;
    __syncthreads();
    const int jn = n - t0 < T ? (int)(n - t0) : T;
    const int j1 = (q + 1) * (T / 4) < jn ? (q + 1) * (T / 4) : jn;
#pragma unroll 8
    for (int j = q * (T / 4); j < j1; ++j) {
      const unsigned long long kj = sk[j];
      before += (kj > ki || (kj == ki && t0 + j < i)) ? 1 : 0;
    }
  }
  part[q][ii] = before;
  __syncthreads();
  if (q == 0 && i < n) {
    const int at = part[0][ii] + part[1][ii] + part[2][ii] + part[3][ii];
    kdst[at] = ki;
    vdst[at] = vsrc[i];
  }
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier of a cooperative launch (every block resident): block count
// arrivals per step on one word.  A wait that outlasts its limit (2^24
// polls, seconds) sets FRICC_DEV_TIMEOUT and gives up; the kernel then
// returns, and its result is reported as failed.
__device__ __forceinline__ bool grid_step(unsigned* bar, unsigned target, unsigned* err, int* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    int ok = 1;
    for (unsigned spins = 0; ld_acquire_u32(bar) < target; ++spins)
      if (spins > (1u << 24)) {
        atomicOr(err, FRICC_DEV_TIMEOUT);
        ok = 0;
        break;
      }
    __threadfence();
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

static __global__ void __launch_bounds__(NT) k_sort_coop(unsigned long long* ksrc, unsigned* vsrc,
                                                         unsigned long long* kdst, unsigned* vdst, int R,
                                                         const int64_t* __restrict__ n_dev, unsigned* hist,
                                                         unsigned* bar, unsigned* err, Batch bt) {
  int64_t maxn = 0;
  for (int r = 0; r < R; ++r) {
    const int64_t c = n_dev[r * bt.n_stride];
    maxn = c > maxn ? c : maxn;
  }
  if (maxn <= RANK_MAX) return;  // uniform over the grid
  __shared__ unsigned h[256];
  __shared__ unsigned wc[NT / 32][256];
  __shared__ int64_t sm[33];
  __shared__ int s_ok;
  unsigned lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  const int w = threadIdx.x >> 5;
  unsigned step = 0;
  unsigned long long *ka = ksrc, *kb = kdst;
  unsigned *va = vsrc, *vb = vdst;
  for (int pass = 0; pass < 9; ++pass) {
    const int shift = 8 * pass;
    if (pass == 8) {  // eight passes end in the source arrays: one copy to the destination
      for (int r = 0; r < R; ++r) {
        const int64_t n = n_dev[r * bt.n_stride], o = r * bt.kv_stride;
        if (n <= RANK_MAX) continue;
        for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
          kdst[o + i] = ksrc[o + i];
          vdst[o + i] = vsrc[o + i];
        }
      }
      return;
    }
    // per-tile digit counts, digit-major
    for (int r = 0; r < R; ++r) {
      const int64_t n = n_dev[r * bt.n_stride], nt = fricc_cdiv(n, (int64_t)TILE);
      if (n <= RANK_MAX) continue;
      const unsigned long long* k = ka + r * bt.kv_stride;
      unsigned* hr = hist + r * bt.hist_stride;
      for (int64_t t = blockIdx.x; t < nt; t += gridDim.x) {
        h[threadIdx.x] = 0;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < IPT; ++q) {
          const int64_t i = t * TILE + q * NT + threadIdx.x;
          if (i < n) atomicAdd(&h[(255u - digit(k[i], shift))], 1u);
        }
        __syncthreads();
        hr[(int64_t)threadIdx.x * nt + t] = h[threadIdx.x];
        __syncthreads();
      }
    }
    if (!grid_step(bar, ++step * gridDim.x, err, &s_ok)) return;
    // each digit's counts scanned over tiles; its total at totals[d]
    for (int r = 0; r < R; ++r) {
      const int64_t n = n_dev[r * bt.n_stride], nt = fricc_cdiv(n, (int64_t)TILE);
      if (n <= RANK_MAX) continue;
      unsigned* hr = hist + r * bt.hist_stride;
      for (int d = blockIdx.x; d < 256; d += gridDim.x) {
        unsigned* row = hr + (int64_t)d * nt;
        const int64_t per = fricc_cdiv(nt, 256), b = threadIdx.x * per, e = b + per < nt ? b + per : nt;
        int64_t loc = 0;
        for (int64_t i = b; i < e; ++i) loc += row[i];
        int64_t tot;
        int64_t run = block_excl_sum(loc, sm, &tot);
        for (int64_t i = b; i < e; ++i) {
          const unsigned c = row[i];
          row[i] = (unsigned)run;
          run += c;
        }
        if (threadIdx.x == 0) hr[256 * nt + d] = (unsigned)tot;
      }
    }
    if (!grid_step(bar, ++step * gridDim.x, err, &s_ok)) return;
    // stable scatter
    for (int r = 0; r < R; ++r) {
      const int64_t n = n_dev[r * bt.n_stride], nt = fricc_cdiv(n, (int64_t)TILE), o = r * bt.kv_stride;
      if (n <= RANK_MAX) continue;
      const unsigned* hr = hist + r * bt.hist_stride;
      int64_t tot;
      const unsigned base = (unsigned)block_excl_sum(hr[256 * nt + threadIdx.x], sm, &tot);
      for (int64_t t = blockIdx.x; t < nt; t += gridDim.x) {
        __syncthreads();
        h[threadIdx.x] = base + hr[(int64_t)threadIdx.x * nt + t];
        for (int q = 0; q < IPT; ++q) {
#pragma unroll
          for (int k = 0; k < NT / 32; ++k) wc[k][threadIdx.x] = 0;
          __syncthreads();
          const int64_t i = t * TILE + q * NT + threadIdx.x;
          const bool valid = i < n;
          const unsigned long long key = valid ? ka[o + i] : 0ull;
          const unsigned val = valid ? va[o + i] : 0u;
          const unsigned d = valid ? (255u - digit(key, shift)) : 256u;
          const unsigned peers = __match_any_sync(0xffffffffu, d);
          const unsigned lrank = __popc(peers & lt);
          if (valid && lrank == 0) wc[w][d] = __popc(peers);
          __syncthreads();
          unsigned acc = h[threadIdx.x];
#pragma unroll
          for (int k = 0; k < NT / 32; ++k) {
            const unsigned c = wc[k][threadIdx.x];
            wc[k][threadIdx.x] = acc;
            acc += c;
          }
          h[threadIdx.x] = acc;
          __syncthreads();
          if (valid) {
            const unsigned pos = wc[w][d] + lrank;
            kb[o + pos] = key;
            vb[o + pos] = val;
          }
          __syncthreads();
        }
      }
    }
    if (!grid_step(bar, ++step * gridDim.x, err, &s_ok)) return;
    unsigned long long* tk = ka;
    ka = kb;
    kb = tk;
    unsigned* tv = va;
    va = vb;
    vb = tv;
  }
}

// (kdst, vdst) = the *n_dev <= n pairs of (ksrc, vsrc) by descending key,
// ties in source order (the source is scratch).  hist: hist_words(n) words
// per replica; bar: one zeroed word; err: an error word.
inline int sort_desc_dev(unsigned long long* ksrc, unsigned* vsrc, unsigned long long* kdst, unsigned* vdst, int64_t n,
                         const int64_t* n_dev, unsigned* hist, unsigned* bar, unsigned* err, cudaStream_t st, int R,
                         Batch bt) {
  const int64_t most = n < RANK_MAX ? n : RANK_MAX;
  k_rank_sort<<<dim3((unsigned)fricc_cdiv(most, RANK_I), (unsigned)R), 256, 0, st>>>(ksrc, vsrc, kdst, vdst, n_dev, bt);
  fricc_note_launch();
  FRICC_LAUNCH_CHECK();
  if (n <= RANK_MAX) return FRICC_OK;
  int dev = 0, nsm = 0, per = 0;
  FRICC_CUDA(cudaGetDevice(&dev));
  FRICC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  FRICC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sort_coop, NT, 0));
  const int64_t tiles = R * fricc_cdiv(n, TILE);
  int64_t g = (int64_t)nsm * (per < 2 ? per : 2);  // two blocks a SM: more would lengthen the barriers
  if (g > tiles) g = tiles;
  void* args[] = {&ksrc, &vsrc, &kdst, &vdst, &R, &n_dev, &hist, &bar, &err, &bt};
  FRICC_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_sort_coop), dim3((unsigned)g), dim3(NT), args,
                                         0, st));
  fricc_note_launch();
  return FRICC_OK;
}

}  // namespace radix
