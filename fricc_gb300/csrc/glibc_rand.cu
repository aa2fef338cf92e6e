// The reference's random stream, generated on the device.
//
// fri-cc draws its uniforms as rand() / RAND_MAX from glibc (src/fri_utils.cpp:47
// for systematic sampling, :73 once per element for pivotal sampling).  glibc's
// default generator (TYPE_3) is an additive lagged-Fibonacci recurrence on
// 32-bit words,
//     r_k = r_{k-31} + r_{k-3}  (mod 2^32),   rand() = r_k >> 1,
// so its whole state is the history h = (r_{k-31}, ..., r_{k-1}) before the
// next draw.  Advancing the history by one draw is a fixed 31x31 linear map M
// over Z/2^32; by C draws it is J = M^C, built on the host by repeated
// squaring.  One block squares J up to the number of chunks, a warp per chunk
// takes the powers of its number's binary digits to its start h_{cC} = J^c h_0,
// and one thread per chunk produces its C words from there, the ring of 31 words
// held in registers (the loop is unrolled 31 deep so every ring index is
// static).  The history after the last draw goes back to the caller, so a
// host-side copy of the stream continues exactly where the device stopped.
#include <vector>

#include "common.cuh"

namespace {

constexpr int RDEG = 31;
constexpr int RSEP = 3;
// Draws per chunk (a multiple of the ring length).  With the starts one after
// another and 1984 draws each, the 549081 draws of o13v57 took 50 us of starts and
// 51 of draws; now 17 (the powers), 9 and 8.
constexpr int64_t GCH = 31 * 8;

// P[b][s * 31 + t] = J^(2^b)[t][s] for b < nb; 1024 threads
__global__ void __launch_bounds__(1024) k_glibc_powers(const unsigned* __restrict__ J, int nb, unsigned* __restrict__ P) {
  __shared__ unsigned A[RDEG * RDEG];
  const int i = threadIdx.x, t = i / RDEG, s = i - t * RDEG;
  const bool in = i < RDEG * RDEG;
  if (in) A[i] = J[i];
  for (int b = 0; b < nb; ++b) {
    __syncthreads();
    unsigned x = 0;
    if (in) {
      P[b * RDEG * RDEG + s * RDEG + t] = A[i];
#pragma unroll
      for (int q = 0; q < RDEG; ++q) x += A[t * RDEG + q] * A[q * RDEG + s];  // wraps mod 2^32
    }
    __syncthreads();
    if (in) A[i] = x;
  }
}

// starts[c * 31 + t] = history at the start of chunk c (oldest first)
__global__ void __launch_bounds__(256) k_glibc_starts(const unsigned* __restrict__ P, const unsigned* __restrict__ h0,
                                                      int64_t nch, unsigned* __restrict__ starts) {
  const int lane = threadIdx.x & 31, t = lane < RDEG ? lane : 0;
  for (int64_t c = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); c < nch; c += (int64_t)gridDim.x * 8) {
    unsigned h = h0[t];
    const unsigned* m = P;
    for (int64_t q = c; q; q >>= 1, m += RDEG * RDEG)
      if (q & 1) {
        unsigned x = 0;
#pragma unroll
        for (int s = 0; s < RDEG; ++s) x += __ldg(m + s * RDEG + t) * __shfl_sync(0xffffffffu, h, s);
        h = x;
      }
    if (lane < RDEG) starts[c * RDEG + lane] = h;
  }
}

// chunk c: draws [c*GCH, min((c+1)*GCH, k)); the thread holding the last draw
// writes the history that follows it
// (the words only: the FP64 division of each draw, in the same thread, made a
// draw ~370 ns, 0.73 ms a chunk; k_glibc_uniform divides in parallel)
__global__ void k_glibc_gen(const unsigned* __restrict__ starts, int64_t nch, int64_t k, unsigned* __restrict__ out,
                            unsigned* __restrict__ hist_out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nch) return;
  unsigned r[RDEG];
#pragma unroll
  for (int t = 0; t < RDEG; ++t) r[t] = starts[c * RDEG + t];
  const int64_t base = c * GCH;
  const int64_t cnt = k - base < GCH ? k - base : GCH;  // > 0
  int64_t done = 0;
  // ring: after d draws of a round the oldest word sits at index d
  while (done < cnt) {
#pragma unroll
    for (int d = 0; d < RDEG; ++d) {
      if (done + d < cnt) {
        const unsigned w = r[d] + r[(d + RDEG - RSEP) % RDEG];
        r[d] = w;
        out[base + done + d] = w;
      }
    }
    done += RDEG;
  }
  if (base + cnt == k) {
    // cnt draws leave the oldest word at ring index cnt % 31
    const int off = (int)(cnt % RDEG);
#pragma unroll
    for (int t = 0; t < RDEG; ++t) hist_out[t >= off ? t - off : t - off + RDEG] = r[t];  // (static ring indices)
  }
}

__global__ void k_glibc_uniform(const unsigned* __restrict__ w, int64_t k, double* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)(int)(w[i] >> 1) / 2147483647.0;
}

using Mat = std::vector<unsigned>;

Mat mat_mul(const Mat& A, const Mat& B) {
  Mat C(RDEG * RDEG, 0u);
  for (int i = 0; i < RDEG; ++i)
    for (int k = 0; k < RDEG; ++k) {
      const unsigned a = A[i * RDEG + k];
      if (!a) continue;
      for (int j = 0; j < RDEG; ++j) C[i * RDEG + j] += a * B[k * RDEG + j];
    }
  return C;
}

// M^e: M maps (h_0..h_30) to (h_1, ..., h_30, h_0 + h_28)
Mat step_power(int64_t e) {
  Mat M(RDEG * RDEG, 0u), R(RDEG * RDEG, 0u);
  for (int t = 0; t + 1 < RDEG; ++t) M[t * RDEG + t + 1] = 1u;
  M[(RDEG - 1) * RDEG + 0] = 1u;
  M[(RDEG - 1) * RDEG + (RDEG - RSEP)] = 1u;
  for (int t = 0; t < RDEG; ++t) R[t * RDEG + t] = 1u;
  while (e > 0) {
    if (e & 1) R = mat_mul(R, M);
    M = mat_mul(M, M);
    e >>= 1;
  }
  return R;
}

}  // namespace

// k uniforms rand()/RAND_MAX of the glibc stream whose history is hist[31]
// (host, oldest first) into out (device); hist is advanced past them.
// Synchronises the stream (the new history is read back).
int fricc_glibc_uniforms_device(unsigned* hist, int64_t k, double* out, cudaStream_t st) {
  if (!hist || k < 0 || (k > 0 && !out)) {
    fricc_set_error("glibc_uniforms: bad arguments");
    return FRICC_ERR_ARG;
  }
  if (k == 0) return FRICC_OK;
  const int64_t nch = fricc_cdiv(k, GCH);
  static const Mat J = step_power(GCH);
  unsigned *dJ = nullptr, *dh = nullptr, *starts = nullptr, *words = nullptr;
  int nb = 0;  // bits of the last chunk's number
  while ((nch - 1) >> nb) ++nb;
  int rc = fricc_alloc_t(&dJ, (size_t)(1 + nb) * RDEG * RDEG + 2 * RDEG, st);
  if (!rc) rc = fricc_alloc_t(&starts, nch * RDEG, st);
  if (!rc) rc = fricc_alloc_t(&words, k, st);
  if (rc) {
    fricc_free(dJ, st);
    fricc_free(starts, st);
    return rc;
  }
  unsigned* const powers = dJ + RDEG * RDEG;
  dh = powers + (size_t)nb * RDEG * RDEG;
  unsigned* dout = dh + RDEG;
  // pageable sources: the copies complete before cudaMemcpyAsync returns
  cudaError_t e = cudaMemcpyAsync(dJ, J.data(), sizeof(unsigned) * RDEG * RDEG, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(dh, hist, sizeof(unsigned) * RDEG, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    const int64_t gs = fricc_cdiv(nch, 8);
    k_glibc_powers<<<1, 1024, 0, st>>>(dJ, nb, powers);
    k_glibc_starts<<<(unsigned)(gs < 152 * 8 ? gs : 152 * 8), 256, 0, st>>>(powers, dh, nch, starts);
    k_glibc_gen<<<(unsigned)fricc_cdiv(nch, 32), 32, 0, st>>>(starts, nch, k, words, dout);
    const int64_t g = fricc_cdiv(k, 256);
    k_glibc_uniform<<<(unsigned)(g < 152 * 16 ? g : 152 * 16), 256, 0, st>>>(words, k, out);
    fricc_note_launch(4);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(hist, dout, sizeof(unsigned) * RDEG, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  fricc_free(starts, st);
  fricc_free(words, st);
  fricc_free(dJ, st);
  return e == cudaSuccess ? FRICC_OK : fricc_cuda_fail(e, "glibc_uniforms", __FILE__, __LINE__);
}
