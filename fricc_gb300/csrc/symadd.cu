// Fused symmetrised accumulation of the T2 residual:
//   out[i,j,a,b] += coef * (X[i,j,a,b] + X[j,i,b,a])
// for X any strided 4-index view (fricc/friccsd.py:245-267 builds these as
// "tmp + tmp.transpose(1,0,3,2)" and adds them to t2new).  out[i,j,a,b] and
// out[j,i,b,a] receive the same sum, so a CTA takes a pair i <= j and a
// 32 x 32 tile of (a,b), reads the two tiles of X once, each along whichever of
// its (a,b) indices is contiguous (through a shared-memory transpose), and
// updates both outputs, the second along its own rows.  All of a thread's loads
// are under way before the first use.  Bound by its bytes: 24 an element; with
// one output per CTA, X was read twice (64 M elements 535 us, now 273).
#include <cstdlib>

#include "common.cuh"

namespace {

constexpr int TD = 32, TR = 8, NR = TD / TR;  // 32 x 32 tile, 32 x 8 threads

struct TileLoad {
  double v[NR];
};
// the tile x(a0 + a', b0 + b') of the plane at `base`: row r of the registers is
// read along b (a' = ty + TR r, b' = tx) or along a (a' = tx, b' = ty + TR r)
__device__ __forceinline__ TileLoad load_tile(const double* __restrict__ X, int64_t base, int64_t sa, int64_t sb, int64_t a0,
                                              int64_t b0, int64_t nv, bool along_b) {
  TileLoad t;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int64_t a = a0 + (along_b ? ty + TR * r : tx), b = b0 + (along_b ? tx : ty + TR * r);
    t.v[r] = (a < nv && b < nv) ? __ldg(X + base + a * sa + b * sb) : 0.0;
  }
  return t;
}
__device__ __forceinline__ void put_tile(double (*tile)[TD + 1], const TileLoad& t, bool along_b) {
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (along_b) tile[ty + TR * r][tx] = t.v[r];
    else tile[tx][ty + TR * r] = t.v[r];
  }
}

__global__ void __launch_bounds__(TD* TR) k_symadd(double* __restrict__ out, const double* __restrict__ X, int64_t o,
                                                    int64_t v, int64_t s0, int64_t s1, int64_t s2, int64_t s3,
                                                    double coef, int first_along_b, int second_along_b,
                                                    int64_t xr = 0) {
  __shared__ double t1[TD][TD + 1], t2[TD][TD + 1];
  // replica batches: blockIdx.z = r o (o + 1) / 2 + pair; replica r's X starts
  // xr elements after the previous one's, its output o^2 v^2 after
  const unsigned np = (unsigned)(o * (o + 1) / 2);  // blockIdx.z < 65536: 32-bit divisions
  const unsigned rep = blockIdx.z / np, pair = blockIdx.z - rep * np;
  X += rep * xr;
  out += rep * o * o * v * v;
  unsigned j = (unsigned)((sqrtf(8.0f * (float)pair + 1.0f) - 1.0f) * 0.5f);  // j (j + 1) / 2 <= pair
  while (j * (j + 1) / 2 > pair) --j;
  while ((j + 1) * (j + 2) / 2 <= pair) ++j;
  const int64_t i = pair - j * (j + 1) / 2;
  const int64_t a0 = (int64_t)blockIdx.y * TD, b0 = (int64_t)blockIdx.x * TD;
  // X[i,j,a,b] over (a,b): strides (s2, s3); X[j,i,b,a] over (a,b): strides (s3, s2)
  const TileLoad x1 = load_tile(X, i * s0 + j * s1, s2, s3, a0, b0, v, first_along_b != 0);
  const TileLoad x2 = load_tile(X, j * s0 + i * s1, s3, s2, a0, b0, v, second_along_b != 0);
  double* o1 = out + ((i * o + j) * v) * v;  // [a][b]
  double* o2 = out + ((j * o + i) * v) * v;  // [b][a]
  const int tx = threadIdx.x, ty = threadIdx.y;
  const bool two = i != (int64_t)j;
  double y1[NR], y2[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int64_t q = ty + TR * r;
    y1[r] = (a0 + q < v && b0 + tx < v) ? o1[(a0 + q) * v + b0 + tx] : 0.0;
    y2[r] = (two && b0 + q < v && a0 + tx < v) ? o2[(b0 + q) * v + a0 + tx] : 0.0;
  }
  put_tile(t1, x1, first_along_b != 0);
  put_tile(t2, x2, second_along_b != 0);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int q = ty + TR * r;
    const double s = t1[q][tx] + t2[q][tx];
    if (a0 + q < v && b0 + tx < v) o1[(a0 + q) * v + b0 + tx] = y1[r] + coef * s;
    t1[q][tx] = s;
  }
  if (!two) return;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int q = ty + TR * r;
    if (b0 + q < v && a0 + tx < v) o2[(b0 + q) * v + a0 + tx] = y2[r] + coef * t1[tx][q];
  }
}

}  // namespace

extern "C" int fricc_symadd(double* out, const double* X, int64_t nocc, int64_t nvir, const int64_t strides[4],
                            double coef, void* stream) {
  if (!out || !X || !strides || nocc <= 0 || nvir <= 0) {
    fricc_set_error("symadd: bad arguments");
    return FRICC_ERR_ARG;
  }
  if (nocc * nocc > 65535) {
    fricc_set_error("symadd: nocc^2 above the grid limit");
    return FRICC_ERR_ARG;
  }
  const int64_t s0 = strides[0], s1 = strides[1], s2 = strides[2], s3 = strides[3];
  // the first read walks (a,b) with strides (s2, s3), the second with (s3, s2)
  const int first_along_b = std::llabs(s3) <= std::llabs(s2) ? 1 : 0;
  const int second_along_b = std::llabs(s2) <= std::llabs(s3) ? 1 : 0;
  const dim3 grid((unsigned)fricc_cdiv(nvir, TD), (unsigned)fricc_cdiv(nvir, TD), (unsigned)(nocc * (nocc + 1) / 2));
  k_symadd<<<grid, dim3(TD, TR), 0, (cudaStream_t)stream>>>(out, X, nocc, nvir, s0, s1, s2, s3, coef, first_along_b,
                                                           second_along_b);
  fricc_note_launch();
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FRICC_OK : fricc_cuda_fail(e, "symadd", __FILE__, __LINE__);
}

// R replicas: out [R][o][o][v][v] (C order), X replica r at X + r xr with
// the per-replica strides of fricc_symadd.
extern "C" int fricc_symadd_b(double* out, const double* X, int64_t R, int64_t nocc, int64_t nvir,
                              const int64_t strides[5], double coef, void* stream) {
  if (!out || !X || !strides || nocc <= 0 || nvir <= 0 || R < 1) {
    fricc_set_error("symadd_b: bad arguments");
    return FRICC_ERR_ARG;
  }
  if (R * nocc * nocc > 65535) {
    fricc_set_error("symadd_b: replicas x nocc^2 above the grid limit");
    return FRICC_ERR_ARG;
  }
  const int64_t s0 = strides[1], s1 = strides[2], s2 = strides[3], s3 = strides[4];
  const int first_along_b = std::llabs(s3) <= std::llabs(s2) ? 1 : 0;
  const int second_along_b = std::llabs(s2) <= std::llabs(s3) ? 1 : 0;
  const dim3 grid((unsigned)fricc_cdiv(nvir, TD), (unsigned)fricc_cdiv(nvir, TD), (unsigned)(R * (nocc * (nocc + 1) / 2)));
  k_symadd<<<grid, dim3(TD, TR), 0, (cudaStream_t)stream>>>(out, X, nocc, nvir, s0, s1, s2, s3, coef, first_along_b,
                                                           second_along_b, strides[0]);
  fricc_note_launch();
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FRICC_OK : fricc_cuda_fail(e, "symadd_b", __FILE__, __LINE__);
}
