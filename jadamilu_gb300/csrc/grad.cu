// Eigenvalue gradients with respect to the stored entries of a sparse
// symmetric matrix (the adjoint / "backward" entry point).
//
// For a simple eigenpair of A x = lambda B x with x^T B x = 1 and B fixed,
// the Hellmann-Feynman theorem gives d lambda / d a_ij = x_i x_j.  A stored
// off-diagonal entry of the one-triangle CSR stands for both a_ij and a_ji,
// so its derivative is 2 x_i x_j.  For f = sum_k w_k lambda_k the gradient is
// the weighted sum over the eigenpairs; for a cluster of equal eigenvalues it
// is basis-independent when the whole cluster is included with one weight.
//
// Device work: per-column normalisation s_k = x_k^T B x_k (B diagonal or I) by
// a deterministic reduction, then one pass over the nonzeros (thread per row,
// rows read their entries and the eigenvector rows once).  X may come column by
// column or row by row: the kernels read either, so no caller has to transpose.
//
// Bound: the copies from and to the caller's arrays (28 MB at n = 260100 and
// six pairs, 0.2 ms at 150 GB/s) and one allocation.  Nine allocations, a column at
// a time in the normalisation and a transposition of C-order eigenvectors on
// the host made it 2.8 ms a call, now 0.63 ms (GB300).
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "../../include/jadamilu_gb300.h"

namespace jdg {
namespace {

constexpr int GR_TPB = 256;
constexpr int GR_MAXK = 64;
constexpr int GR_CH = 8;  // columns a thread carries at once

// coef[c] = w_c / sum_i bdiag_i x_c(i)^2; X(i, c) at i * rs + c * cs.  Every CTA
// writes its partial sums, the last to arrive (count starts at zero) adds them
// in CTA order: strided over 32 lanes, then the warp tree.
__global__ void __launch_bounds__(GR_TPB) colnorm_kernel(int n, int k, const double* __restrict__ X, long rs, long cs,
                                                         const double* __restrict__ bdiag,
                                                         const double* __restrict__ w, double* partial,
                                                         unsigned* count, double* __restrict__ coef) {
  __shared__ double red[GR_TPB / 32][GR_CH];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nb = gridDim.x;
  for (int c0 = 0; c0 < k; c0 += GR_CH) {
    double s[GR_CH] = {};
    for (int i = blockIdx.x * GR_TPB + threadIdx.x; i < n; i += nb * GR_TPB) {
      const double b = bdiag ? bdiag[i] : 1.0;
#pragma unroll
      for (int c = 0; c < GR_CH; ++c)
        if (c0 + c < k) {
          const double v = X[i * rs + (c0 + c) * cs];
          s[c] += b * v * v;
        }
    }
#pragma unroll
    for (int c = 0; c < GR_CH; ++c) {
      for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
      if (lane == 0) red[wid][c] = s[c];
    }
    __syncthreads();
    if (threadIdx.x < GR_CH && c0 + threadIdx.x < k) {
      double t = 0;
      for (int q = 0; q < GR_TPB / 32; ++q) t += red[q][threadIdx.x];
      partial[(long)(c0 + threadIdx.x) * nb + blockIdx.x] = t;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(count, 1u) == (unsigned)nb - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  for (int c = wid; c < k; c += GR_TPB / 32) {
    double t = 0;
    for (int b = lane; b < nb; b += 32) t += __ldcg(partial + (long)c * nb + b);
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) coef[c] = w[c] / t;
  }
}

// grad[q] = c_q * sum_c coef_c x_c(i) x_c(j), i the row of stored entry q; KM
// columns in registers.  A row pointer or column out of range sets *bad.
template <int KM>
__global__ void __launch_bounds__(GR_TPB) eig_grad_kernel(int n, int nnz, int k, const int* __restrict__ ia,
                                                          const int* __restrict__ ja, const double* __restrict__ X,
                                                          long rs, long cs, const double* __restrict__ coef,
                                                          double* __restrict__ grad, unsigned* bad) {
  const int i = blockIdx.x * GR_TPB + threadIdx.x;
  if (i >= n) return;
  double xi[KM];
#pragma unroll
  for (int c = 0; c < KM; ++c) xi[c] = c < k ? coef[c] * X[i * rs + c * cs] : 0.0;
  const int b = ia[i] - 1, e = ia[i + 1] - 1;
  if (b < 0 || e > nnz) {
    *bad = 1;
    return;
  }
  for (int q = b; q < e; ++q) {
    const int j = ja[q] - 1;
    if (j < 0 || j >= n) {
      *bad = 1;
      continue;
    }
    double g = 0;
#pragma unroll
    for (int c = 0; c < KM; ++c)
      if (c < k) g += xi[c] * X[j * rs + c * cs];
    grad[q] = (j == i) ? g : 2.0 * g;
  }
}

int eig_grad(int n, const int* ia, const int* ja, int neig, const double* X, long rs, long cs, long xlen,
             const double* w, const double* bdiag, double* grad) {
  const int nnz = ia[n] - 1;
  if (nnz < 0) return -1;
  unsigned char* base = nullptr;
  int rc = 0;
  try {
    const int nb = std::min(std::max(1, (n + GR_TPB - 1) / GR_TPB), 152 * 4);
    size_t used = 0;
    auto place = [&](size_t bytes) {
      const size_t at = used;
      used += (bytes + 255) / 256 * 256;
      return at;
    };
    const size_t oia = place(sizeof(int) * ((size_t)n + 1)), oja = place(sizeof(int) * (size_t)std::max(1, nnz)),
                 oX = place(sizeof(double) * (size_t)xlen), ow = place(sizeof(double) * neig),
                 ob = place(bdiag ? sizeof(double) * (size_t)n : 0), op = place(sizeof(double) * (size_t)nb * neig),
                 oc = place(sizeof(double) * neig), of = place(2 * sizeof(unsigned)),
                 og = place(sizeof(double) * (size_t)std::max(1, nnz));
    CK(cudaMalloc(&base, used));
    int *dia = (int*)(base + oia), *dja = (int*)(base + oja);
    double *dX = (double*)(base + oX), *dw = (double*)(base + ow), *db = bdiag ? (double*)(base + ob) : nullptr,
           *dpart = (double*)(base + op), *dcoef = (double*)(base + oc), *dg = (double*)(base + og);
    unsigned* flags = (unsigned*)(base + of);  // arrival counter, out-of-range flag
    const cudaStream_t st = nullptr;
    CK(cudaMemsetAsync(flags, 0, 2 * sizeof(unsigned), st));
    CK(cudaMemcpyAsync(dX, X, sizeof(double) * (size_t)xlen, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dw, w, sizeof(double) * neig, cudaMemcpyHostToDevice, st));
    if (bdiag) CK(cudaMemcpyAsync(db, bdiag, sizeof(double) * n, cudaMemcpyHostToDevice, st));
    colnorm_kernel<<<nb, GR_TPB, 0, st>>>(n, neig, dX, rs, cs, db, dw, dpart, flags, dcoef);
    CK(cudaMemcpyAsync(dia, ia, sizeof(int) * ((size_t)n + 1), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dja, ja, sizeof(int) * (size_t)nnz, cudaMemcpyHostToDevice, st));
    const dim3 g((n + GR_TPB - 1) / GR_TPB);
    auto go = [&](auto kern) { kern<<<g, GR_TPB, 0, st>>>(n, nnz, neig, dia, dja, dX, rs, cs, dcoef, dg, flags + 1); };
    if (neig <= 8) go(eig_grad_kernel<8>);
    else if (neig <= 16) go(eig_grad_kernel<16>);
    else go(eig_grad_kernel<GR_MAXK>);
    CK(cudaGetLastError());
    k::add_launches(2);
    unsigned bad = 0;
    CK(cudaMemcpyAsync(&bad, flags + 1, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(grad, dg, sizeof(double) * (size_t)nnz, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (bad) rc = -1;
  } catch (std::exception& e) {
    std::fprintf(stderr, "jdgpu_deig_grad: %s\n", e.what());
    rc = -99;
  }
  cudaFree(base);
  return rc;
}

}  // namespace
}  // namespace jdg

using namespace jdg;

// Gradient of sum_k w[k] lambda_k with respect to every stored entry of the
// one-triangle CSR (ia, ja) used for A; see include/jadamilu_gb300.h.
JDG_API int jdgpu_deig_grad(int n, const int* ia, const int* ja, int neig, const double* X, int ldx,
                            const double* w, const double* bdiag, double* grad) {
  if (n <= 0 || neig <= 0 || neig > GR_MAXK || ldx < n) return -1;
  return eig_grad(n, ia, ja, neig, X, 1, ldx, (long)ldx * (neig - 1) + n, w, bdiag, grad);
}
JDG_API int jdgpu_deig_grad_rows(int n, const int* ia, const int* ja, int neig, const double* X, const double* w,
                                 const double* bdiag, double* grad) {
  if (n <= 0 || neig <= 0 || neig > GR_MAXK) return -1;
  return eig_grad(n, ia, ja, neig, X, neig, 1, (long)n * neig, w, bdiag, grad);
}
