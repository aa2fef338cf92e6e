// FP64-accurate matrix products on the tensor cores by modular integer
// arithmetic (gemm_mod.cu): what the FP64 GEMM and sparse-term dispatches use.
#pragma once
#include "common.cuh"

// Element (r) of a row index that flattens up to three levels
// r = (i2 * n1 + i1) * n0 + i0, at i2 s2 + i1 s1 + i0 s0 (element strides).
struct ModRows {
  int64_t n2 = 1, n1 = 1, n0 = 1;
  int64_t s2 = 0, s1 = 0, s0 = 0;
  int64_t off = 0;  // the first row of a panel
  // a level outside the current ones (which it therefore sweeps slowest)
  void outer(int64_t n, int64_t s) {
    if (n == 1) return;
    if (n0 == 1 && n1 == 1 && n2 == 1) {
      n0 = n;
      s0 = s;
    } else if (n1 == 1 && n2 == 1) {
      n1 = n;
      s1 = s;
    } else {
      n2 = n;
      s2 = s;
    }
  }
  __device__ __forceinline__ int64_t at(int64_t r) const {
    r += off;
    if (n1 == 1 && n2 == 1) return r * s0;
    const int64_t q = r / n0, i0 = r - q * n0;
    const int64_t i2 = q / n1, i1 = q - i2 * n1;
    return i2 * s2 + i1 * s1 + i0 * s0;
  }
};

// One operand: rows x K, element (r, k) at x + rows.at(r) + k * sk, or, with
// kn > 0 (a contraction index of two levels), (k / kn) * sko + (k % kn) * sk.
// With `prepared`, the buffer fricc_mod_operand filled from exactly these rows.
struct ModView {
  const double* x = nullptr;
  ModRows rows;
  int64_t sk = 0;
  int64_t kn = 0, sko = 0;
  const void* prepared = nullptr;
  __device__ __forceinline__ int64_t kat(int64_t k) const {
    if (kn == 0) return k * sk;
    const int64_t q = (int64_t)((unsigned)k / (unsigned)kn);  // k < 2^22
    return q * sko + (k - q * kn) * sk;
  }
};

// C[rep][r][c] = alpha sum_k A[rep][r][k] B[rep][c][k] + beta C, element
// (rep, r, c) of C at C + rep.at(rep) + row.at(r) + col.at(c).
struct ModOut {
  double* C = nullptr;
  ModRows row, col, rep;
  double alpha = 1.0, beta = 0.0;
};

// A and B hold reps * M and (b_shared ? N : reps * N) rows, replica-major (A
// likewise with a_shared).  skip_zero: elements of A whose bits are all
// zero are absent (they multiply nothing, not even a NaN of B).
// FRICC_MOD_NONE: its scratch could not be had (or it is too large for a
// launch), and nothing was written.
constexpr int FRICC_MOD_NONE = -1;
int fricc_mod_gemm(const ModView& A, const ModView& B, const ModOut& out, int64_t M, int64_t N, int64_t K, int64_t reps,
                   bool a_shared, bool b_shared, bool skip_zero, cudaStream_t st);

// Estimated time (us) of fricc_mod_gemm; conv_a / conv_b: whether the
// operand is still to be converted.
double fricc_mod_time_us(int64_t M, int64_t N, int64_t K, int64_t reps, bool a_shared, bool b_shared, bool conv_a,
                         bool conv_b);

// Bytes of a prepared operand of `rows` x k, and its preparation.
int64_t fricc_mod_operand_bytes(int64_t rows, int64_t k);
int fricc_mod_operand(const ModView& v, int64_t rows, int64_t k, void* buf, cudaStream_t st);

// Estimates (us) of a batched product on the FP64 (or FP32-pair) GEMM
// kernels, and the choice: the modular product where its estimate is below
// 0.8 of `alt_us`.
double fricc_mod_alt_us(int64_t batch, int64_t M, int64_t N, int64_t K, bool pairs);
bool fricc_mod_chosen(int64_t batch, int64_t M, int64_t N, int64_t K, bool a_batched, bool b_batched, bool a_prepared,
                      bool b_prepared, double alt_us);

// C = alpha A B + beta C of the strided batched GEMMs (fricc_gemm_f64's
// arguments; s2: the second batch level's strides or null) through
// fricc_mod_gemm where that is chosen over the caller's kernel (FP64, or
// FP32 pairs).  The choice does not depend on the second batch level, so a
// replica takes the route of its lone product.  Returns a status, or
// FRICC_MOD_NONE when not taken.
int fricc_mod_try(const double* A, const double* B, double* C, int64_t batch, int64_t batch2, int64_t M, int64_t N,
                  int64_t K, const int64_t sA[3], const int64_t sB[3], const int64_t sC[3], const int64_t* s2,
                  double alpha, double beta, bool pairs, const void* a_mod, const void* b_mod, cudaStream_t st);
