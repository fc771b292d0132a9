// Jacobi-Davidson core on device vectors (host control, sm_103a kernels).
//
// Same algorithm as the reference's JDRVCOM/LSOLREVCOM/STOPTEST/REPGS/
// SOLPROJEP/SHRINK/SORTEV (src/jd/JDaux.F:1391-3358).  Every N-length vector
// lives on the GPU in `dX`, a device copy of the caller's workspace X with the
// reference layout (JDaux.F:1534-1567), so reverse-communication offsets
// (NDX1/NDX2/NDX3) and the eigenvector output keep their meaning.  The J x J
// projected matrices and the small coefficient vectors stay in the caller's
// host X at the same offsets.  Scalars that steer the control flow (norms,
// inner products) are written to pinned host words by the kernels that form
// them; the host watches those words (DevJd::await).
#pragma once
#include <cfloat>
#include <chrono>
#include <complex>
#include <functional>
#include <vector>

#include "kernels.cuh"
#include "small_dense.hpp"

namespace jdg {

template <class T> struct HostOf { using type = double; };
template <> struct HostOf<zc> { using type = std::complex<double>; };
inline double hre(double x) { return x; }
inline double hre(std::complex<double> x) { return x.real(); }
inline double habs(double x) { return std::fabs(x); }
inline double habs(std::complex<double> x) { return std::abs(x); }
inline double tod(double x) { return x; }
inline zc todev(std::complex<double> x) { return zc(x.real(), x.imag()); }
inline double todev(double x) { return x; }

// values shared with the preconditioner-aware driver (COMMON /JDRVCOMJD/)
struct JdState {
  double timeilu = 0, rinit = 0, rcurr = 0, rcum = 0, shift1 = 0;
  bool flagcg = false;
};

// Device workspace of one solve.
template <class T> struct Workspace {
  cudaStream_t st = nullptr;
  long N = 0, LX = 0, cap_x = 0, cap_tmp = 0, cap_part = 0;
  T* dX = nullptr;     // device copy of X
  T* dsm = nullptr;    // small device results (<= 512)
  T* hsm = nullptr;    // pinned host mirror
  T* dpart = nullptr;  // reduction partials
  T* dtmp = nullptr;   // N x 32 scratch for restarts
  // the one-launch inner iteration: partial sums it leaves for the host, its
  // grid barrier's counter and what the host knows it holds
  double* hpart = nullptr;
  unsigned* dbar = nullptr;
  k::OneState one;
  void reset_barrier() {
    CK(cudaMemsetAsync(dbar, 0, sizeof(unsigned), st));
    one.base = 0;
  }
  bool own_stream = false;
  // Every entry leaves its stream idle (Idle), so a caller's stream needs no wait here
  void set_stream(cudaStream_t s) {
    if (own_stream && st) {
      cudaStreamSynchronize(st);
      cudaStreamDestroy(st);
    }
    st = s;
    own_stream = false;
  }
  void ensure(long n, long lx) {
    if (!st) {
      CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
      own_stream = true;
    }
    if (!dsm) {
      CK(cudaMalloc(&dsm, sizeof(T) * 512));
      CK(cudaMallocHost(&hsm, sizeof(T) * 512));
      CK(cudaMallocHost(&hpart, sizeof(double) * k::kMaxPartials));
      CK(cudaMalloc(&dbar, sizeof(unsigned)));
      reset_barrier();
    }
    if (lx > cap_x) {
      if (dX) CK(cudaFree(dX));
      CK(cudaMalloc(&dX, sizeof(T) * lx));
      cap_x = lx;
    }
    long need_tmp = n * 32;
    if (need_tmp > cap_tmp) {
      if (dtmp) CK(cudaFree(dtmp));
      CK(cudaMalloc(&dtmp, sizeof(T) * need_tmp));
      cap_tmp = need_tmp;
    }
    long need_part = k::mdot_partial_size(n, 128);
    if (need_part > cap_part) {
      if (dpart) CK(cudaFree(dpart));
      CK(cudaMalloc(&dpart, sizeof(T) * need_part));
      CK(cudaMemset(dpart, 0, sizeof(T) * need_part));  // the reduction's arrival counter starts at zero
      cap_part = need_part;
    }
    N = n;
    LX = lx;
  }
  // frees everything (the workspace of a batch worker ends with its thread)
  void release() {
    if (dX) cudaFree(dX);
    if (dsm) cudaFree(dsm);
    if (hsm) cudaFreeHost(hsm);
    if (hpart) cudaFreeHost(hpart);
    if (dbar) cudaFree(dbar);
    if (dpart) cudaFree(dpart);
    if (dtmp) cudaFree(dtmp);
    if (own_stream && st) cudaStreamDestroy(st);
    dX = dsm = hsm = dpart = dtmp = nullptr;
    hpart = nullptr;
    dbar = nullptr;
    st = nullptr;
    own_stream = false;
    cap_x = cap_tmp = cap_part = 0;
  }
  ~Workspace() {}
};

// Waits for the workspace's stream at the end of a scope, exceptions included: a
// kernel still in flight could write host words that the next solve watches,
// or work on buffers that it hands to another stream.
template <class T> struct Idle {
  Workspace<T>& W;
  ~Idle() {
    if (W.st) cudaStreamSynchronize(W.st);
  }
};

template <class T> struct StopStateD {
  int istag = 0, istt = 0;
  bool posdef = false, toupdate = false;
  double g0 = 0, gs = 0, gtrs = 0, gkmin = 0, bk = 0, beta = 0, tn = 0, un2 = -1, gkm1 = 0, alp = 1;
  typename HostOf<T>::type bkgep = 0, bubt = 0;
};

struct Lcg48d {
  unsigned long long s = 0x1234ABCD330EULL;
  double next() {
    s = (s * 0x5DEECE66DULL + 0xB) & ((1ULL << 48) - 1);
    return ((double)(s >> 5) + 0.5) / (double)(1ULL << 43);
  }
};

template <class T> struct DevJd {
  using H = typename HostOf<T>::type;
  Workspace<T>* W = nullptr;
  JdState* sh = nullptr;
  H* hX = nullptr;  // caller's X (small J x J data live here)
  // which: 1 = A x (and B x for GEP), 3 = A x, 4 = B x; offsets into X
  std::function<void(int, long, long, long)> matvec;
  std::function<void(long, long)> precond;  // (rhs, sol)
  // built-in matrix: y = A x + a x (GEP: yb = B x, y = A x + a yb) in one kernel (offsets x, y, yb)
  std::function<void(long, long, long, double)> matvec_shift;
  // built-in matrix: the whole inner iteration outside the preconditioner in
  // one launch (k columns from U and BU; offsets z, r, p), see k::inner_one
  std::function<int(int, long, long, long, long, long, double, bool, bool, T*, const T*)> inner_one;
  std::function<void(int, int, int, double, double)> on_step;  // progress printer (may be empty)
  StopStateD<T> st;
  Lcg48d rng;
  double alpha_cg = 0;
  int istag = 0;
  long launches = 0;
  // The operators are the library's own stream-ordered kernels (no host
  // round trip inside matvec/precond): the inner iteration may then keep its
  // scalars on the device and read them back once per iteration.
  bool device_ops = false;
  static constexpr int kScal = 500;  // dsm / hsm slots of the inner-iteration scalars
  static constexpr int kCoef = 320;  // hsm slots of a projection's coefficients (64), read later
  static constexpr int kLate = 400;  // hsm slot of an inner product read later

  T* D(long off) { return W->dX + off; }
  cudaStream_t S() { return W->st; }
  void sync() { CK(cudaStreamSynchronize(S())); }

  // A kernel whose results the host needs writes them into the pinned mirror
  // itself.  The host marks those words before the launch and watches them
  // instead of waiting for the stream: 2 us less per read (9 us from launch to
  // wake-up on GB300).  After kWatch (long kernels before it, an error, a value
  // with the mark's bits) it waits for the stream after all; await returns
  // whether all words were written then.
  static constexpr unsigned long long kMark = 0x7FF4DEADBEEF5A5AULL;  // a signalling NaN no kernel produces
  static constexpr std::chrono::microseconds kWatch{300};
  template <class V> static void mark(V* h, long n) {
    auto* w = reinterpret_cast<unsigned long long*>(h);
    for (long i = 0; i < n * (long)(sizeof(V) / 8); ++i) __atomic_store_n(w + i, kMark, __ATOMIC_RELEASE);
  }
  template <class V> bool await(const V* h, long n) {
    const auto* w = reinterpret_cast<const unsigned long long*>(h);
    const long words = n * (long)(sizeof(V) / 8);
    const auto until = std::chrono::steady_clock::now() + kWatch;
    for (long i = 0; i < words; ++i)
      for (int t = 1; __atomic_load_n(w + i, __ATOMIC_ACQUIRE) == kMark; ++t)
        if (t % 256 == 0 && std::chrono::steady_clock::now() > until) {
          sync();
          for (; i < words; ++i)
            if (__atomic_load_n(w + i, __ATOMIC_ACQUIRE) == kMark) return false;
          return true;
        }
    return true;
  }

  // ---- device primitives on X offsets ----
  double nrm2(long n, long x) {
    mark(W->hsm, 1);
    k::mdot<T>(n, 1, D(x), n, D(x), W->hsm, W->dpart, S());
    await(W->hsm, 1);
    return std::sqrt(rl(W->hsm[0]));
  }
  H dot(long n, long x, long y) {
    mark(W->hsm, 1);
    k::mdot<T>(n, 1, D(x), n, D(y), W->hsm, W->dpart, S());
    await(W->hsm, 1);
    return reinterpret_cast<H*>(W->hsm)[0];
  }
  // out_host[c] = X(V + c*ldv)^H X(w), c < k
  void gemvc(long n, int kc, long V, long ldv, long w, H* out_host) {
    if (kc <= 0) return;
    for (int c0 = 0; c0 < kc; c0 += 128) {
      int kk = std::min(128, kc - c0);
      mark(W->hsm, kk);
      k::mdot<T>(n, kk, D(V + (long)c0 * ldv), ldv, D(w), W->hsm, W->dpart, S());
      await(W->hsm, kk);
      for (int c = 0; c < kk; ++c) out_host[c0 + c] = reinterpret_cast<H*>(W->hsm)[c];
    }
  }
  // two of them with the same vector, read together (at most 64 columns each)
  void gemvc2(long n, int kc, long V, long V2, long ldv, long w, H* out, H* out2) {
    if (kc > 64) {
      gemvc(n, kc, V, ldv, w, out);
      gemvc(n, kc, V2, ldv, w, out2);
      return;
    }
    mark(W->hsm, 64 + kc);
    k::mdot<T>(n, kc, D(V), ldv, D(w), W->hsm, W->dpart, S());
    k::mdot<T>(n, kc, D(V2), ldv, D(w), W->hsm + 64, W->dpart, S());
    await(W->hsm, kc);
    await(W->hsm + 64, kc);
    const H* h = reinterpret_cast<const H*>(W->hsm);
    for (int c = 0; c < kc; ++c) {
      out[c] = h[c];
      out2[c] = h[64 + c];
    }
  }
  // X(w) = beta X(w) + alpha X(V) y, y on the host
  void gemvn(long n, int kc, double alpha, long V, long ldv, const H* y, double beta, long w) {
    std::vector<T> yd(std::max(kc, 1));
    for (int c = 0; c < kc; ++c) yd[c] = todev(y[c]);
    for (int c0 = 0; c0 < std::max(kc, 1); c0 += 64) {
      int kk = std::min(64, kc - c0);
      const double b = (c0 == 0) ? beta : 1.0;
      k::gemv_val<T>(n, std::max(kk, 0), alpha, D(V + (long)c0 * ldv), ldv, yd.data() + c0, b, D(w), S());
      if (kc <= 0) break;
    }
  }
  void axpy(long n, H a, long x, long y) { k::axpy<T>(n, todev(a), D(x), D(y), S()); }
  void scal(long n, double a, long x) { k::scal<T>(n, a, D(x), S()); }
  void copy(long n, long x, long y) {
    if (n > 0 && x != y) CK(cudaMemcpyAsync(D(y), D(x), sizeof(T) * n, cudaMemcpyDeviceToDevice, S()));
  }
  void fill(long n, H v, long x) { k::fill<T>(n, todev(v), D(x), S()); }

  // REPGS on device vectors; y (coefficients and final norm) on the host
  void repgs(long N, long V, long BV, long JV, long w, H* y, double epsm, int gam) {
    bool nrnd = true;
    if (JV <= 0) return;
    if (gam < 0) {
      // classical Gram-Schmidt, coefficients stay on the device; y, when
      // given, asks for them on the host (repgs_coef)
      if (JV > 64) throw std::runtime_error("projection against more than 64 vectors");
      if (y) mark(W->hsm + kCoef, JV);
      k::mdot<T>(N, (int)JV, D(BV), N, D(w), W->dsm, W->dpart, S());
      k::gemv_dev<T>(N, (int)JV, -1.0, D(V), N, W->dsm, 1.0, D(w), S(), y ? W->hsm + kCoef : nullptr);
      return;
    }
    // up to 63 columns: a pass leaves its coefficients on the device between
    // the inner products and the update, which also gives the new norm (and
    // the first pass takes the old norm as one more column), and is read back
    // once
    const bool one_read = JV < 64;
    for (;;) {
      double nrn = one_read ? 0.0 : nrm2(N, w), nr = epsm * nrn, nro;
      if (nrnd)
        for (long c = 0; c < JV; ++c) y[c] = H(0);
      bool small = false, first = true;
      do {
        nro = nrn;
        if (one_read) {
          mark(W->hsm, JV + 2);
          k::mdot<T>(N, (int)JV + first, D(BV), N, D(w), W->dsm, W->dpart, S(), first ? D(w) : nullptr);
          k::gemv_dot<T>(N, (int)JV, D(V), N, W->dsm, D(w), nullptr, W->dsm + JV + 1, W->dpart, S(), W->dsm,
                         (int)JV + 2, W->hsm);
          await(W->hsm, JV + 2);
          const H* h = reinterpret_cast<const H*>(W->hsm);
          for (long c = 0; c < JV; ++c) y[JV + c] = h[c];
          if (first) {
            nro = std::sqrt(rl(W->hsm[JV]));
            nr = epsm * nro;
          }
          nrn = std::sqrt(rl(W->hsm[JV + 1]));
          first = false;
        } else {
          gemvc(N, (int)JV, BV, N, w, y + JV);
          gemvn(N, (int)JV, -1.0, V, N, y + JV, 1.0, w);
          nrn = nrm2(N, w);
        }
        if (nrnd)
          for (long c = 0; c < JV; ++c) y[c] += y[JV + c];
        if (nrn <= nr) { small = true; break; }
      } while (nrn < 0.5 * nro);
      if (!small) { y[JV] = H(nrn); return; }
      if (gam == 1) {
        if (JV < N) {
          std::vector<T> r(N);
          for (long i = 0; i < N; ++i) r[i] = T(rng.next());
          CK(cudaMemcpyAsync(D(w), r.data(), sizeof(T) * N, cudaMemcpyHostToDevice, S()));
          sync();
          nrnd = false;
          continue;
        }
      } else {
        fill(N, H(0), w);
        y[JV] = H(0);
      }
      return;
    }
  }

  // coefficient c of the last projection with gam < 0
  H repgs_coef(long c) {
    await(W->hsm + kCoef + c, 1);
    return reinterpret_cast<const H*>(W->hsm)[kCoef + c];
  }

  // SORTEV on host arrays (small) or device columns (eigenvectors)
  void sort_index_key(long J, const double* eigs, int it, double sigma, std::vector<long>& iw) {
    std::vector<double> key(J);
    for (long i = 0; i < J; ++i) {
      if (it == 2 || it == -2) key[i] = -std::fabs(eigs[i] - sigma);
      else if (it == 4 || it == -4) key[i] = eigs[i];
      else key[i] = -eigs[i];
    }
    iw.resize(J);
    jdd::sort_index(J, key.data(), iw.data());
    if (it == -2) {
      long last = iw[J - 1];
      for (long i = J - 1; i > 0; --i) iw[i] = iw[i - 1];
      iw[0] = last;
    }
  }
  void sortev_host(long J, H* V, long ldv, double* eigs, int it) {
    if (J <= 1) return;
    std::vector<long> iw;
    sort_index_key(J, eigs, it, 0.0, iw);
    std::vector<H> tv(J * J);
    for (long c = 0; c < J; ++c)
      for (long r = 0; r < J; ++r) tv[r + c * J] = V[r + iw[c] * ldv];
    for (long c = 0; c < J; ++c)
      for (long r = 0; r < J; ++r) V[r + c * ldv] = tv[r + c * J];
    std::vector<double> te(J);
    for (long c = 0; c < J; ++c) te[c] = eigs[iw[c]];
    for (long c = 0; c < J; ++c) eigs[c] = te[c];
  }
  void sortev_dev(long N, long J, long V, long V2, double* eigs, double* r, int it, double sigma) {
    if (J <= 1) return;
    std::vector<long> iw;
    sort_index_key(J, eigs, it, sigma, iw);
    auto permute = [&](long base) {
      for (long c = 0; c < J; ++c)
        CK(cudaMemcpyAsync(W->dtmp + c * N, D(base + iw[c] * N), sizeof(T) * N, cudaMemcpyDeviceToDevice, S()));
      CK(cudaMemcpyAsync(D(base), W->dtmp, sizeof(T) * N * J, cudaMemcpyDeviceToDevice, S()));
    };
    if (J > 32) throw std::runtime_error("sortev: more than 32 vectors");
    permute(V);
    if (it == -4) permute(V2);
    std::vector<double> te(J);
    for (long c = 0; c < J; ++c) te[c] = eigs[iw[c]];
    for (long c = 0; c < J; ++c) eigs[c] = te[c];
    if (it == 4 || it == -4) {
      for (long c = 0; c < J; ++c) te[c] = r[iw[c]];
      for (long c = 0; c < J; ++c) r[c] = te[c];
    }
  }
  // SOLPROJEP (JDaux.F:3271-3358); the generalized harmonic case solves
  // NN X = MM (POSV) and takes the right eigenvectors of X (GEEV).
  void solprojep(long J, H* MM, H* NN, long ld, double& theta, double& theta2, double* w, int is, int& info, bool gep) {
    if (is == 2 || is == -2) {
      if (gep) {
        info = jdd::posv_u(J, NN, ld, MM, ld);
        if (info) return;
        jdd::copyv(ld * ld, MM, NN);
        info = jdd::geev_right(J, NN, ld, w, MM, ld);
        if (info) return;
        sortev_host(J, MM, ld, w, is);
        theta2 = w[1];
        return;
      }
      info = jdd::hegv(J, MM, ld, NN, ld, w);
      if (info) return;
      sortev_host(J, MM, ld, w, is);
      theta2 = w[1];
      return;
    }
    jdd::herm_full(J, MM, ld);
    info = jdd::heev(J, MM, ld, w);
    if (info) return;
    if (is == 3) {
      for (long i = 0; i < J; ++i) NN[i] = H(w[i]);
    } else {
      theta = w[0];
      theta2 = w[1];
    }
  }
  void shrink(long N, long J, long K, const H* U, long ldu, long V, long Wv, long BV, H* MM, H* NN, long ld,
              int iserch, bool gep) {
    if (K > 32) throw std::runtime_error("shrink: search space above 32");
    std::vector<H> Q;
    jdd::householder_q(K, J, U, ldu, Q);
    std::vector<T> qd(K * K);
    for (long i = 0; i < K * K; ++i) qd[i] = todev(Q[i]);
    auto apply = [&](long base) {
      k::rmult<T>(N, (int)K, (int)J, D(base), N, qd.data(), W->dtmp, S());
      CK(cudaMemcpyAsync(D(base), W->dtmp, sizeof(T) * N * J, cudaMemcpyDeviceToDevice, S()));
    };
    apply(V);
    apply(Wv);
    if (gep) apply(BV);
    auto congr = [&](H* M, bool herm) {
      if (herm)
        for (long i = 1; i < K; ++i)
          for (long j = 0; j < i; ++j) M[i + j * ld] = jdd::cj(M[j + i * ld]);
      std::vector<H> tmp(K * K), out(K * K);
      for (long j = 0; j < K; ++j)
        for (long i = 0; i < K; ++i) {
          H s = H(0);
          for (long kk = 0; kk < K; ++kk) s += M[i + kk * ld] * Q[kk + j * K];
          tmp[i + j * K] = s;
        }
      for (long j = 0; j < K; ++j)
        for (long i = 0; i < K; ++i) {
          H s = H(0);
          for (long kk = 0; kk < K; ++kk) s += jdd::cj(Q[kk + i * K]) * tmp[kk + j * K];
          out[i + j * K] = s;
        }
      for (long j = 0; j < K; ++j)
        for (long i = 0; i < K; ++i) M[i + j * ld] = out[i + j * K];
    };
    congr(MM, iserch != 2 || !gep);
    if (iserch == 2) congr(NN, true);
  }
  void stoptest(long N, long x, long bt, long bu, double tol, double& rk, double nbu, double& alprho, double& gk,
                H pcad, H pcr, double& theta, double eta, int& info, double trs, bool gep);
  void run(long N, double* EIGS, double* RES, int LX, int& NEIG, double SIGMA, int ISEARCH, int NINIT, int MADSPACE,
           int& ITER, double TOL, int& INFO, double& GAP, bool GEP);
};

}  // namespace jdg
