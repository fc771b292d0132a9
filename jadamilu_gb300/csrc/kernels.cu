// sm_103a kernels of the Jacobi-Davidson hot path.
//
// All of them are HBM-bandwidth kernels (no tensor-core work exists on this
// path): SpMV over the full Hermitian matrix in SELL-32 layout (coalesced
// column/value loads), the level-scheduled sweeps of the multilevel LDL^H
// preconditioner, and the BLAS-1/2 vector work of the outer and inner JD
// iterations (deterministic reductions, so results do not depend on timing).
// Short problems are bound by launches and dependent latencies instead, float64
// ones also by the FP64 units; each kernel says which.
#include <algorithm>
#include <atomic>
#include <climits>
#include <functional>
#include <map>
#include <type_traits>

#include <mutex>

#include <cooperative_groups.h>

#include "kernels.cuh"

namespace jdg {
namespace k {

static std::atomic<long long> g_launches{0};
long long launch_count() { return g_launches.load(); }
void add_launches(long long n) { g_launches += n; }
#define COUNT_LAUNCH() (g_launches += 1)

constexpr int TPB = 256;

// Programmatic dependent launch inside the preconditioner graph: a kernel
// lets its successor be scheduled as soon as all of its CTAs have started
// (launch_dependents), and waits for its predecessor to complete and flush
// (griddepcontrol.wait) before reading anything.  Both are no-ops for a
// kernel launched without the attribute.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The two halves of pdl_begin, for kernels that load data before waiting for
// the predecessor's results: those loads overlap the predecessor's tail.  They
// are ordered after no kernel of the stream but those complete at its last full
// ordering point (a synchronisation, a copy, a launch without the attribute): a
// predecessor that released its successor at its start may itself still wait for
// the kernel before it.  So they may touch only data that is finished before
// the kernels that read it are launched: the factor (upload_factor ends in a
// synchronisation), the matrix (build_sell does) and its slice pointers.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Asks the TMA unit to bring [p, p + bytes) into L2 and returns at once (a
// hint: nothing waits for it or reads it back).  Only the 16-byte aligned
// interior of the range is requested, in pieces of at most 64 KB, so no byte
// outside [p, p + bytes) is touched.
__device__ __forceinline__ void l2_prefetch(const void* p, size_t bytes) {
  size_t a = __cvta_generic_to_global(p);
  size_t e = a + bytes;
  a = (a + 15) & ~(size_t)15;
  e &= ~(size_t)15;
  while (a < e) {
    const unsigned sz = (unsigned)(e - a < 65536 ? e - a : 65536);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(sz) : "memory");
    a += sz;
  }
}
static bool g_pdl = true;
void set_pdl(bool on) { g_pdl = on; }
template <class... Params, class... Args>
static void launch_k(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = g_pdl ? 1 : 0;
  CK(cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...));
}
static inline int nblk(long n, int tpb = TPB) { return (int)std::max<long>(1, (n + tpb - 1) / tpb); }

// ---------------------------------------------------------------- SpMV ----
// The first kSellPre entries of a row (SELL-32: entry j of a slice's row at
// 32 j + lane) are loaded before waiting for the predecessor that writes x,
// then gathered together and added in entry order, as one at a time.
constexpr int kSellPre = 8;
template <class T> struct SellBatch {
  int c[kSellPre];
  T v[kSellPre];
};
template <class T>
__device__ __forceinline__ void sell_load(SellBatch<T>& b, int64_t q, int64_t e, const int* __restrict__ col,
                                          const T* __restrict__ val) {
#pragma unroll
  for (int u = 0; u < kSellPre; ++u) {
    const int64_t qq = q + 32 * u;
    if (qq < e) {
      b.c[u] = __ldg(col + qq);
      b.v[u] = val[qq];
    } else {
      b.c[u] = -1;
      b.v[u] = T(0);
    }
  }
}
template <class T> __device__ __forceinline__ T sell_use(const SellBatch<T>& b, const T* __restrict__ x, T acc) {
  T w[kSellPre];
#pragma unroll
  for (int u = 0; u < kSellPre; ++u) w[u] = b.c[u] >= 0 ? x[b.c[u]] : T(0);
#pragma unroll
  for (int u = 0; u < kSellPre; ++u)
    if (b.c[u] >= 0) acc = fma_(b.v[u], w[u], acc);
  return acc;
}
template <class T>
__global__ void __launch_bounds__(TPB) spmv_sell_kernel(int n, const int64_t* __restrict__ sptr,
                                                        const int* __restrict__ col, const T* __restrict__ val,
                                                        const T* __restrict__ x, T* __restrict__ y) {
  pdl_launch();
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  int sl = r >> 5, lane = r & 31;
  int64_t b = sptr[sl], e = sptr[sl + 1];
  SellBatch<T> first;
  sell_load(first, b + lane, e, col, val);
  pdl_wait();
  T acc = sell_use(first, x, T(0));
  for (int64_t q = b + lane + kSellPre * 32; q < e; q += 32) acc = fma_(val[q], x[__ldg(col + q)], acc);
  y[r] = acc;
}
template <class T> void spmv(const SellMatrix<T>& A, const T* x, T* y, cudaStream_t s) {
  launch_k(spmv_sell_kernel<T>, dim3(nblk(A.n)), dim3(TPB), 0, s, A.n, A.sptr, A.col, A.val, x, y);
  COUNT_LAUNCH();
}
// ------------------------------------------- SELL-32 from one triangle ----
// The full Hermitian matrix in SELL-32, built on the device from the caller's
// one-triangle CSR (1-based).  A row's entries are ordered as a host pass over
// the stored entries would append them: by the row they are stored in, then by
// position; so transposed entries (i, p) of rows before it, its own, those of
// rows after it (the other triangle).
//   sell_count   transposed entries per row, row and index checks
//   sell_width   full row lengths, slice widths, totals
//   sell_scan    slice pointers
//   sell_fill    every off-diagonal entry's key (i, p) into a slot of its
//                column's row, in any order
//   sell_finish  a row's keys sorted, columns and values written, padding
// Bound: the copy of the triangle to the device and the memory it writes; the
// host pass took 2 ms at n = 64000 and 33 ms at n = 1e6 (GB300's Grace).  A product
// through the public call, hand-over included: n = 125000 4.0 -> 0.61 ms.
constexpr int kSellKeys = 64;     // most transposed entries per row (more: the host pass)
constexpr int kSellOwn = 4096;    // most stored entries per row
// info: 0 stored slots, 1 full nonzeros, 2 a bad row pointer or column, 3 a row beyond the limits above
__global__ void __launch_bounds__(TPB) sell_count_kernel(int n, int nnz, const int* __restrict__ ia,
                                                         const int* __restrict__ ja, int* __restrict__ tcnt,
                                                         unsigned long long* __restrict__ info) {
  pdl_begin();
  const int i = blockIdx.x * TPB + threadIdx.x;
  if (i >= n) return;
  const int b = ia[i] - 1, e = ia[i + 1] - 1;
  if (b < 0 || e < b || e > nnz) {
    atomicOr(info + 2, 1ull);
    return;
  }
  if (e - b > kSellOwn) {
    atomicOr(info + 3, 1ull);
    return;
  }
  for (int p = b; p < e; ++p) {
    const int j = ja[p] - 1;
    if (j < 0 || j >= n) atomicOr(info + 2, 1ull);
    else if (j != i && atomicAdd(tcnt + j, 1) >= kSellKeys) atomicOr(info + 3, 1ull);
  }
}
__global__ void __launch_bounds__(TPB) sell_width_kernel(int n, const int* __restrict__ ia, const int* __restrict__ tcnt,
                                                         int64_t* __restrict__ sptr,
                                                         unsigned long long* __restrict__ info) {
  pdl_begin();
  const int r = blockIdx.x * TPB + threadIdx.x, lane = threadIdx.x & 31;
  const int cnt = r < n ? ia[r + 1] - ia[r] + tcnt[r] : 0;
  const int w = __reduce_max_sync(0xffffffffu, cnt < 0 ? 0 : cnt);
  const unsigned sum = __reduce_add_sync(0xffffffffu, (unsigned)(cnt < 0 ? 0 : cnt));
  if (lane == 0 && (r >> 5) < (n + 31) / 32) {
    sptr[(r >> 5) + 1] = (int64_t)w * 32;
    atomicAdd(info + 1, (unsigned long long)sum);
  }
}
// in-place inclusive scan of sptr[1..ns] by one CTA; sptr[0] = 0, info[0] = the total
constexpr int kScanTpb = 1024;
__global__ void __launch_bounds__(kScanTpb) sell_scan_kernel(int ns, int64_t* __restrict__ sptr,
                                                             unsigned long long* __restrict__ info) {
  pdl_begin();
  __shared__ int64_t part[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t done = 0;
  for (int s0 = 0; s0 < ns; s0 += kScanTpb) {
    const int s = s0 + threadIdx.x;
    int64_t v = s < ns ? sptr[s + 1] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    if (lane == 31) part[wid] = v;
    __syncthreads();
    int64_t before = done, all = done;
    for (int w = 0; w < 32; ++w) {
      if (w < wid) before += part[w];
      all += part[w];
    }
    if (s < ns) sptr[s + 1] = before + v;
    done = all;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    sptr[0] = 0;
    info[0] = (unsigned long long)done;
  }
}
template <class T>
__global__ void __launch_bounds__(TPB) sell_fill_kernel(int n, const int* __restrict__ ia, const int* __restrict__ ja,
                                                        const int64_t* __restrict__ sptr, int* __restrict__ cur,
                                                        T* __restrict__ val) {
  pdl_begin();
  const int i = blockIdx.x * TPB + threadIdx.x;
  if (i >= n) return;
  for (int p = ia[i] - 1; p < ia[i + 1] - 1; ++p) {
    const int j = ja[p] - 1;
    if (j == i) continue;
    const int k = atomicAdd(cur + j, 1);
    *reinterpret_cast<unsigned long long*>(val + sptr[j >> 5] + (int64_t)k * 32 + (j & 31)) =
        ((unsigned long long)(unsigned)i << 32) | (unsigned)p;
  }
}
template <class T>
__global__ void __launch_bounds__(TPB) sell_finish_kernel(int n, const int* __restrict__ ia, const int* __restrict__ ja,
                                                          const T* __restrict__ a, const int64_t* __restrict__ sptr,
                                                          const int* __restrict__ tcnt, int* __restrict__ col,
                                                          T* __restrict__ val) {
  pdl_begin();
  const int r = blockIdx.x * TPB + threadIdx.x, lane = r & 31, s = r >> 5;
  if (s >= (n + 31) / 32) return;
  const int64_t at = sptr[s] + lane;
  const int width = (int)((sptr[s + 1] - sptr[s]) / 32);
  int q = 0;
  auto put = [&](int c, T v) {
    col[at + (int64_t)q * 32] = c;
    val[at + (int64_t)q * 32] = v;
    ++q;
  };
  if (r < n) {
    const int nt = tcnt[r];
    unsigned long long key[kSellKeys];
    for (int k = 0; k < nt; ++k) {  // insertion sort: rows have a handful
      const unsigned long long v = *reinterpret_cast<const unsigned long long*>(val + at + (int64_t)k * 32);
      int h = k;
      for (; h > 0 && key[h - 1] > v; --h) key[h] = key[h - 1];
      key[h] = v;
    }
    int k = 0;
    auto transposed = [&](int below) {  // the keys of rows before `below`
      for (; k < nt && (int)(key[k] >> 32) < below; ++k) put((int)(key[k] >> 32), cj(a[(unsigned)key[k]]));
    };
    transposed(r);
    for (int p = ia[r] - 1; p < ia[r + 1] - 1; ++p) put(ja[p] - 1, a[p]);
    transposed(n);
  }
  const int c = r < n ? r : 0;
  while (q < width) put(c, T(0));
}
static int64_t round256(int64_t b) { return (b + 255) / 256 * 256; }
int64_t sell_work_bytes(int n, int64_t nnz, int64_t value) {
  return round256(4 * (int64_t)(n + 1)) + round256(4 * nnz) + round256(value * nnz) + 2 * round256(4 * (int64_t)n) +
         round256(8 * 4);
}
template <class T>
bool sell_from_triangle(int n, const int* ia, const int* ja, const void* a, void* work, int64_t* sptr,
                        unsigned long long* info_host, const std::function<void(int64_t, int**, T**)>& room,
                        cudaStream_t s) {
  const int nnz = ia[n] - 1;
  unsigned char* w = (unsigned char*)work;
  auto take = [&](int64_t bytes) {
    unsigned char* p = w;
    w += round256(bytes);
    return (void*)p;
  };
  int* dia = (int*)take(4 * (int64_t)(n + 1));
  int* dja = (int*)take(4 * (int64_t)nnz);
  T* da = (T*)take(sizeof(T) * (int64_t)nnz);
  int* tcnt = (int*)take(4 * (int64_t)n);
  int* cur = (int*)take(4 * (int64_t)n);
  unsigned long long* info = (unsigned long long*)take(8 * 4);
  CK(cudaMemsetAsync(tcnt, 0, (unsigned char*)info + 32 - (unsigned char*)tcnt, s));
  CK(cudaMemcpyAsync(dia, ia, 4 * (size_t)(n + 1), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(dja, ja, 4 * (size_t)nnz, cudaMemcpyHostToDevice, s));
  const dim3 g(nblk(n)), t(TPB);
  launch_k(sell_count_kernel, g, t, 0, s, n, nnz, dia, dja, tcnt, info);
  launch_k(sell_width_kernel, g, t, 0, s, n, dia, tcnt, sptr, info);
  launch_k(sell_scan_kernel, dim3(1), dim3(kScanTpb), 0, s, (n + 31) / 32, sptr, info);
  CK(cudaMemcpyAsync(info_host, info, 8 * 4, cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(da, a, sizeof(T) * (size_t)nnz, cudaMemcpyHostToDevice, s));
  CK(cudaStreamSynchronize(s));
  if (info_host[2]) throw std::runtime_error("row pointers or column indices out of range");
  if (info_host[3]) return false;
  int* col = nullptr;
  T* val = nullptr;
  room((int64_t)info_host[0], &col, &val);
  // the caller synchronises before a product reads what these write (see pdl_launch)
  launch_k(sell_fill_kernel<T>, g, t, 0, s, n, dia, dja, sptr, cur, val);
  launch_k(sell_finish_kernel<T>, g, t, 0, s, n, dia, dja, da, sptr, tcnt, col, val);
  g_launches += 5;
  return true;
}

// -------------------------------------------------------------- BLAS-1 ----
// Complex vectors times real scalars: the products with a zero imaginary part,
// which cannot change a sum, are left out.  FP64 instructions are the bound of
// the complex kernels from about 1e5 rows on (2 FMA per SM and cycle).
__device__ __forceinline__ double axpy_re(double a, double x, double y) { return fma(a, x, y); }
__device__ __forceinline__ zc axpy_re(double a, zc x, zc y) { return zc(fma(a, x.x, y.x), fma(a, x.y, y.y)); }
__device__ __forceinline__ double im_(double) { return 0.0; }
__device__ __forceinline__ double im_(zc a) { return a.y; }
template <class T> __global__ void axpy_kernel(long n, T a, const T* __restrict__ x, T* __restrict__ y) {
  pdl_begin();
  const bool real = im_(a) == 0.0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = real ? axpy_re(rl(a), x[i], y[i]) : fma_(a, x[i], y[i]);
}
// y -= (Re *c / den) x with *c in device memory (the result of an earlier reduction)
template <class T>
__global__ void axpy_dev_kernel(long n, const T* c, double den, const T* __restrict__ x, T* __restrict__ y) {
  pdl_begin();
  const double a = den == 1 ? -rl(*c) : -rl(*c) / den;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = axpy_re(a, x[i], y[i]);
}
template <class T> __global__ void scal_kernel(long n, double a, T* x) {
  pdl_begin();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) x[i] = a * x[i];
}
template <class T> __global__ void fill_kernel(long n, T v, T* x) {
  pdl_begin();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) x[i] = v;
}
static inline int grid_1d(long n) { return (int)std::min<long>(nblk(n), 152L * 16); }
template <class T> void axpy(long n, T a, const T* x, T* y, cudaStream_t s) {
  if (n > 0) { launch_k(axpy_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, a, x, y); COUNT_LAUNCH(); }
}
template <class T> void axpy_dev(long n, const T* c, double den, const T* x, T* y, cudaStream_t s) {
  if (n > 0) { launch_k(axpy_dev_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, c, den, x, y); COUNT_LAUNCH(); }
}
template <class T> void scal(long n, double a, T* x, cudaStream_t s) {
  if (n > 0) { launch_k(scal_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, a, x); COUNT_LAUNCH(); }
}
template <class T> void fill(long n, T v, T* x, cudaStream_t s) {
  if (n > 0) { launch_k(fill_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, v, x); COUNT_LAUNCH(); }
}

// ---------------------------------------------------- reductions (V^H w) ----
__device__ __forceinline__ float shfl_xor_any(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double shfl_xor_any(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ cc shfl_xor_any(cc v, int o) { return cc(shfl_xor_any(v.x, o), shfl_xor_any(v.y, o)); }
__device__ __forceinline__ zc shfl_xor_any(zc v, int o) { return zc(shfl_xor_any(v.x, o), shfl_xor_any(v.y, o)); }

// loads that bypass L1 (data another CTA of the same launch wrote)
__device__ __forceinline__ double ldcg_(const double* p) { return __ldcg(p); }
__device__ __forceinline__ zc ldcg_(const zc* p) {
  const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
  return zc(v.x, v.y);
}

constexpr int MD_CH = 8;       // most columns that one tree carries
constexpr int MD_GROUPS = 32;  // column groups of one call
constexpr int MD_COLS = 128;   // columns of one call
constexpr int MD_WARPS = TPB / 32;
// Long vectors: up to two rows per thread, enough CTAs in flight to stream V
// at full bandwidth.  Vectors under 4096 rows keep one CTA per 2048 rows, the
// summation order validated on the user-guide samples (n = 1000), whose JD
// trajectories change with the rounding of these inner products.
static inline int md_grid(long n) {
  if (n < 4096) return (int)std::max<long>(1, (n + 2047) / 2048);
  return (int)std::min<long>((n + 511) / 512, kMaxPartials);
}

int reduction_blocks(long n) { return md_grid(n); }

// The partials follow one arrival counter per column group at the start of
// the buffer (zero when the buffer is allocated; the last CTA of a group
// resets its counter).
constexpr int MD_HEAD = MD_GROUPS * (int)sizeof(unsigned);
static_assert(MD_HEAD <= kPartialHead * (int)sizeof(double), "the counters fit before the partials");
long mdot_partial_size(long n, int k) {
  return (long)md_grid(n) * k + kPartialHead;
}

// The warp tree (lane pairs 16, 8, 4, 2, 1 apart) of CH values per lane (CH a
// power of two).  The first steps halve the columns a lane carries instead of
// repeating the whole tree per column (CH = 8: 9 exchanges instead of 40, the
// same pairs added).  The sum of column md_col<CH>(lane) ends in the lanes
// whose lowest bits (lane % (32 / CH)) are zero.
template <class T, int CH> __device__ __forceinline__ T md_tree(T (&v)[CH], int lane) {
  int o = 16;
#pragma unroll
  for (int h = CH / 2; h > 0; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < CH / 2; ++j)
      if (j < h) {
        const T send = up ? v[j] : v[j + h];
        v[j] = (up ? v[j + h] : v[j]) + shfl_xor_any(send, o);
      }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] += shfl_xor_any(v[0], o);
  return v[0];
}
template <int CH> __device__ __forceinline__ int md_col(int lane) {
  static_assert(CH == 1 || CH == 2 || CH == 4 || CH == 8, "column groups of 1, 2, 4 or 8");
  const int b4 = (lane >> 4) & 1, b3 = (lane >> 3) & 1, b2 = (lane >> 2) & 1;
  return CH == 1 ? 0 : CH == 2 ? b4 : CH == 4 ? b4 * 2 + b3 : b4 * 4 + b3 * 2 + b2;
}

// A lane's share of the g partials of nc columns: those at 32 w + lane, step
// TPB, of warp w.  The warp tree of each w, then w in order, completes the sum.
template <class T, int CH>
__device__ __forceinline__ T (*md_partials(const T* p, int nc, int g, int w, int lane, T (&s)[CH]))[CH] {
#pragma unroll
  for (int c = 0; c < CH; ++c) s[c] = T(0);
#pragma unroll 1
  for (int q = 32 * w + lane; q < g; q += TPB)
#pragma unroll
    for (int c = 0; c < CH; ++c)
      if (c < nc) s[c] += ldcg_(p + (long)c * g + q);
  return &s;
}

// The sum of one column's g <= 32 partials by one warp; every lane returns it.
template <class T> __device__ __forceinline__ T md_sum_32(const T* p, int g, int lane) {
  T s[1] = {T(0)};
  if (lane < g) s[0] += ldcg_(p + lane);
  return md_tree(s, lane);
}

// The end of a reduction whose threads hold CH partial sums each: a column's
// sums go up the warp tree, then over the CTA's warps in order; the CTA of the
// group that arrives last (a counter, no waiting) adds the CTAs' partials the
// same way, its threads striding over them, so the result does not depend on
// which CTA is last.  This tail bounds the short reductions (store, fence,
// atomic, loads, and two chains of dependent float64 additions of some 50
// cycles each).  us a call (GB300), one CTA going through the columns one by
// one with two barriers each -> here: one column n = 4096 4.9 -> 4.1, 64000 7.3
// -> 6.9, 1e6 14.9 -> 12.5; 12 to 50 us on average over the solves before.
// Returns true in the CTA that wrote the group's results.
template <class T, int CH>
__device__ __forceinline__ bool md_finish(T (&acc)[CH], int nc, int c0, unsigned char* buf, T* out) {
  __shared__ T red[MD_WARPS][CH];
  __shared__ bool last;
  unsigned* count = reinterpret_cast<unsigned*>(buf) + blockIdx.y;
  T* partial = reinterpret_cast<T*>(buf + MD_HEAD);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = gridDim.x;
  const T v = md_tree(acc, lane);
  if (lane % (32 / CH) == 0) red[wid][md_col<CH>(lane)] = v;
  __syncthreads();
  if (threadIdx.x < nc) {
    T t = T(0);
#pragma unroll
    for (int q = 0; q < MD_WARPS; ++q) t += red[q][threadIdx.x];
    if (g == 1) out[c0 + threadIdx.x] = t;
    else partial[(long)(c0 + threadIdx.x) * g + blockIdx.x] = t;
  }
  if (g == 1) return true;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(count, 1u) == (unsigned)g - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return false;
  if (g <= 32) {  // only warp 0 would find partials: a warp per column, and done
    if (wid < nc) {
      const T t = md_sum_32(partial + (long)(c0 + wid) * g, g, lane);
      if (lane == 0) out[c0 + wid] = t;
    }
  } else {
    T s[CH];
    const T f = md_tree(*md_partials<T, CH>(partial + (long)c0 * g, nc, g, wid, lane, s), lane);
    if (lane % (32 / CH) == 0) red[wid][md_col<CH>(lane)] = f;
    __syncthreads();
    if (threadIdx.x < nc) {
      T t = T(0);
#pragma unroll
      for (int q = 0; q < MD_WARPS; ++q) t += red[q][threadIdx.x];
      out[c0 + threadIdx.x] = t;
    }
  }
  if (threadIdx.x == 0) *count = 0u;
  return true;
}

// Columns per group of mdot: four instead of eight leave registers for more
// resident CTAs, which hide the trees.  us for 25 columns, eight -> four
// (GB300): n = 1e6 136 -> 96.6, 262144 42.3 -> 32.5, 64000 13.5 -> 11.6, complex
// 262144 105 -> 76.2; for five columns at n = 64000 8.0 -> 9.9.
constexpr int MD_GRP = 4;
static_assert(MD_COLS <= MD_GRP * MD_GROUPS, "a counter for every group");

// V^H w in one launch, a grid row of CTAs per group of CH columns.
// xcol, when given, is column k - 1 (a vector that does not follow V's others).
template <class T, int CH>
__global__ void __launch_bounds__(TPB) mdot_kernel(long n, int k, const T* __restrict__ V, long ldv,
                                                   const T* __restrict__ w, const T* __restrict__ xcol,
                                                   unsigned char* __restrict__ buf, T* __restrict__ out) {
  pdl_begin();
  const int c0 = blockIdx.y * CH;
  const int nc = min(CH, k - c0);
  const T* cp[CH];
#pragma unroll
  for (int j = 0; j < CH; ++j) cp[j] = xcol && c0 + j == k - 1 ? xcol : V + (long)(c0 + j) * ldv;
  T acc[CH];
#pragma unroll
  for (int j = 0; j < CH; ++j) acc[j] = T(0);
  // two rows' loads in flight at once, added in row order
  const long step = (long)gridDim.x * TPB;
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += 2 * step) {
    const bool two = i + step < n;
    T v0[CH], v1[CH];
#pragma unroll
    for (int j = 0; j < CH; ++j)
      if (j < nc) {
        v0[j] = cp[j][i];
        v1[j] = two ? cp[j][i + step] : T(0);
      }
    const T w0 = w[i], w1 = two ? w[i + step] : T(0);
#pragma unroll
    for (int j = 0; j < CH; ++j)
      if (j < nc) {
        acc[j] = fma_(cj(v0[j]), w0, acc[j]);
        if (two) acc[j] = fma_(cj(v1[j]), w1, acc[j]);
      }
  }
  md_finish<T, CH>(acc, nc, c0, buf, out);
}
template <class T>
void mdot(long n, int k, const T* V, long ldv, const T* w, T* out, T* partial, cudaStream_t s, const T* xcol) {
  if (k <= 0) return;
  if (k > MD_COLS) throw std::runtime_error("mdot: too many columns");
  unsigned char* buf = reinterpret_cast<unsigned char*>(partial);
  const int g = md_grid(n);
  if (k == 1)
    launch_k(mdot_kernel<T, 1>, dim3(g), dim3(TPB), 0, s, n, k, V, ldv, w, xcol, buf, out);
  else
    launch_k(mdot_kernel<T, MD_GRP>, dim3(g, (k + MD_GRP - 1) / MD_GRP), dim3(TPB), 0, s, n, k, V, ldv, w, xcol,
             buf, out);
  g_launches += 1;
}

// ------------------------------------------------------ V y (tall-skinny) ----
constexpr int GMV_MAX = 64;
constexpr int kColBatch = 4;  // columns of a projection whose loads are in flight at once
template <class T> struct SmallVec { T v[GMV_MAX]; };

template <class T>
__global__ void __launch_bounds__(TPB) jd_basis_gemv_dev_kernel(long n, int k, double alpha, const T* __restrict__ V, long ldv,
                                                       const T* __restrict__ y, double beta, T* __restrict__ w,
                                                       T* __restrict__ hy) {
  pdl_begin();
  __shared__ T ys[GMV_MAX];
  if (threadIdx.x < k) {
    ys[threadIdx.x] = y[threadIdx.x];
    if (hy && blockIdx.x == 0) hy[threadIdx.x] = ys[threadIdx.x];
  }
  __syncthreads();
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += (long)gridDim.x * TPB) {
    T acc = T(0);
    for (int c = 0; c < k; ++c) acc = fma_(V[i + (long)c * ldv], ys[c], acc);
    const T o = beta == 0 ? T(0) : beta == 1 ? w[i] : beta * w[i];
    w[i] = axpy_re(alpha, acc, o);
  }
}
template <class T>
__global__ void __launch_bounds__(TPB) jd_basis_gemv_val_kernel(long n, int k, double alpha, const T* __restrict__ V, long ldv,
                                                       SmallVec<T> y, double beta, T* __restrict__ w) {
  pdl_begin();
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += (long)gridDim.x * TPB) {
    T acc = T(0);
    for (int c = 0; c < k; ++c) acc = fma_(V[i + (long)c * ldv], y.v[c], acc);
    const T o = beta == 0 ? T(0) : beta == 1 ? w[i] : beta * w[i];
    w[i] = axpy_re(alpha, acc, o);
  }
}
template <class T>
void gemv_dev(long n, int k, double alpha, const T* V, long ldv, const T* y, double beta, T* w, cudaStream_t s, T* hy) {
  if (k > GMV_MAX) throw std::runtime_error("gemv_dev: too many columns");
  if (k <= 0) {
    if (beta != 1) {
      if (beta == 0) fill(n, T(0), w, s);
      else throw std::runtime_error("gemv_dev: unsupported beta");
    }
    return;
  }
  launch_k(jd_basis_gemv_dev_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, k, alpha, V, ldv, y, beta, w, hy);
  COUNT_LAUNCH();
}
template <class T>
void gemv_val(long n, int k, double alpha, const T* V, long ldv, const T* yh, double beta, T* w, cudaStream_t s) {
  if (k > GMV_MAX) throw std::runtime_error("gemv_val: too many columns");
  if (k <= 0) {
    if (beta == 0) fill(n, T(0), w, s);
    return;
  }
  SmallVec<T> y;
  for (int c = 0; c < k; ++c) y.v[c] = yh[c];
  launch_k(jd_basis_gemv_val_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, k, alpha, V, ldv, y, beta, w);
  COUNT_LAUNCH();
}

// the real part of acc + conj(a) b, with the roundings of fma_
__device__ __forceinline__ double dot_re(double a, double b, double acc) { return fma(a, b, acc); }
__device__ __forceinline__ double dot_re(zc a, zc b, double acc) { return fma(a.x, b.x, fma(a.y, b.y, acc)); }

// w = w - V y (y in device memory), out[0] = x^H w (x = nullptr: w^H w); then,
// with nsc > 0, the nsc scalars from sc on go to the host's pinned hsc.  ratio,
// when given, is Re out / Re rden, or Re rnum / Re out: the scalar of the
// update that follows.  (Divided there, by every warp, it cost that update
// some 40 FP64 instructions of 16 cycles a warp: n = 262144, direction 13.2
// -> 2.5 us, residual 18.4 -> 10.3 us.)
template <class T>
__global__ void __launch_bounds__(TPB) gemv_dot_kernel(long n, int k, const T* __restrict__ V, long ldv, const T* y,
                                                       T* w, const T* x, unsigned char* buf, T* out, const T* sc,
                                                       int nsc, T* hsc, const T* rnum, const T* rden, double* ratio) {
  pdl_begin();
  __shared__ T ys[GMV_MAX];
  if (threadIdx.x < k) ys[threadIdx.x] = y[threadIdx.x];
  __syncthreads();
  T dot[1] = {T(0)};
  const long step = (long)gridDim.x * TPB;
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += 2 * step) {  // two rows at once, as mdot
    const bool two = i + step < n;
    const long i1 = two ? i + step : i;
    const T o0 = w[i], o1 = w[i1], x0 = x ? x[i] : T(0), x1 = x ? x[i1] : T(0);
    T a0 = T(0), a1 = T(0);
    int c0 = 0;
    for (; c0 + kColBatch <= k; c0 += kColBatch) {  // the loads of a batch first, then its products in order
      T v0[kColBatch], v1[kColBatch];
#pragma unroll
      for (int c = 0; c < kColBatch; ++c) {
        v0[c] = V[i + (long)(c0 + c) * ldv];
        v1[c] = V[i1 + (long)(c0 + c) * ldv];
      }
#pragma unroll
      for (int c = 0; c < kColBatch; ++c) {
        a0 = fma_(v0[c], ys[c0 + c], a0);
        a1 = fma_(v1[c], ys[c0 + c], a1);
      }
    }
#pragma unroll 1
    for (; c0 < k; ++c0) {
      const T v0 = V[i + (long)c0 * ldv], v1 = V[i1 + (long)c0 * ldv];
      a0 = fma_(v0, ys[c0], a0);
      a1 = fma_(v1, ys[c0], a1);
    }
    const T r0 = o0 - a0, r1 = o1 - a1;
    w[i] = r0;
    dot[0] = fma_(cj(x ? x0 : r0), r0, dot[0]);
    if (two) {
      w[i1] = r1;
      dot[0] = fma_(cj(x ? x1 : r1), r1, dot[0]);
    }
  }
  if (!md_finish<T, 1>(dot, 1, 0, buf, out)) return;
  __syncthreads();
  if (threadIdx.x < nsc) hsc[threadIdx.x] = sc[threadIdx.x];
  if (threadIdx.x == 0 && ratio) *ratio = rden ? rl(*out) / rl(*rden) : rl(*rnum) / rl(*out);
}
template <class T>
void gemv_dot(long n, int k, const T* V, long ldv, const T* y, T* w, const T* x, T* out, T* partial, cudaStream_t s,
              const T* sc, int nsc, T* hsc, const T* rnum, const T* rden, double* ratio) {
  if (k < 1 || k > GMV_MAX) throw std::runtime_error("projection against more than 64 vectors");
  auto go = [&](auto kern) {
    launch_k(kern, dim3(md_grid(n)), dim3(TPB), 0, s, n, k, V, ldv, y, w, x, reinterpret_cast<unsigned char*>(partial), out,
             sc, nsc, hsc, rnum, rden, ratio);
  };
  go(gemv_dot_kernel<T>);
  COUNT_LAUNCH();
}

// The search direction: z += *be p and p = z (be = Re rho / Re rho0, from
// gemv_dot); the first iteration (be = nullptr) takes p = z, and leaves p alone when rho ends the
// inner solve (zero, or not positive where the preconditioner should be), since
// p is then its result.
template <class T>
__global__ void __launch_bounds__(TPB) cg_direction_kernel(long n, const T* rho, const double* be, bool posdef, T* p, T* z) {
  pdl_begin();
  if (!be) {
    const double r = rl(*rho);
    if (r == 0 || (posdef && r <= 0)) return;
    for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += (long)gridDim.x * TPB) p[i] = z[i];
    return;
  }
  const double a = *be;
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += (long)gridDim.x * TPB) {
    const T t = axpy_re(a, p[i], z[i]);
    z[i] = t;
    p[i] = t;
  }
}
template <class T>
void cg_direction(long n, const T* rho, const double* be, bool posdef, T* p, T* z, cudaStream_t s) {
  launch_k(cg_direction_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, rho, be, posdef, p, z);
  COUNT_LAUNCH();
}

// y = A x + a x, or with B: yb = B x, y = A x + a yb.  Its inner products are
// left to mdot: a thread per row needs the whole grid in flight, while mdot's
// order gives a thread up to four rows one after another (n = 1e6: 43 us in
// that order, 33 us as two kernels; n = 1000: 6.3 and 4.4 us).
template <class T, bool GEP>
__global__ void __launch_bounds__(TPB) spmv_shift_kernel(int n, const int64_t* __restrict__ sptr,
                                                         const int* __restrict__ col, const T* __restrict__ val,
                                                         const int64_t* __restrict__ bptr, const int* __restrict__ bcol,
                                                         const T* __restrict__ bval, double a, const T* __restrict__ x,
                                                         T* __restrict__ y, T* __restrict__ yb) {
  pdl_launch();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int sl = r >> 5, lane = r & 31;
  const int64_t b = sptr[sl], e = sptr[sl + 1];
  SellBatch<T> first;
  sell_load(first, b + lane, e, col, val);
  pdl_wait();
  T acc = sell_use(first, x, T(0));
  for (int64_t q = b + lane + kSellPre * 32; q < e; q += 32) acc = fma_(val[q], x[__ldg(col + q)], acc);
  T u = x[r];
  if (GEP) {
    const int64_t b2 = bptr[sl], e2 = bptr[sl + 1];
    sell_load(first, b2 + lane, e2, bcol, bval);
    u = sell_use(first, x, T(0));
    for (int64_t q = b2 + lane + kSellPre * 32; q < e2; q += 32) u = fma_(bval[q], x[__ldg(bcol + q)], u);
    yb[r] = u;
  }
  y[r] = axpy_re(a, u, acc);
}
template <class T>
void spmv_shift(const SellMatrix<T>& A, const SellMatrix<T>* B, double a, const T* x, T* y, T* yb, cudaStream_t s) {
  const int64_t* bp = B ? B->sptr : nullptr;
  const int* bc = B ? B->col : nullptr;
  const T* bv = B ? B->val : nullptr;
  auto go = [&](auto kern) {
    launch_k(kern, dim3(nblk(A.n)), dim3(TPB), 0, s, A.n, A.sptr, A.col, A.val, bp, bc, bv, a, x, y, yb);
  };
  if (B) go(spmv_shift_kernel<T, true>);
  else go(spmv_shift_kernel<T, false>);
  COUNT_LAUNCH();
}

// r -= *al q (al = Re rho / Re p^H q, from gemv_dot), out[0] = r^H r; the finishing CTA then copies the
// iteration's nsc scalars (sc, out among them) to the host's pinned hsc.
template <class T>
__global__ void __launch_bounds__(TPB) cg_residual_kernel(long n, const double* al, const T* __restrict__ q,
                                                          T* __restrict__ r, unsigned char* buf, T* out, const T* sc,
                                                          int nsc, T* hsc) {
  pdl_begin();
  const double a = -1.0 * *al;
  T dot[1] = {T(0)};
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += (long)gridDim.x * TPB) {
    const T t = axpy_re(a, q[i], r[i]);
    r[i] = t;
    dot[0] = T(dot_re(t, t, rl(dot[0])));
  }
  if (!md_finish<T, 1>(dot, 1, 0, buf, out)) return;
  __syncthreads();
  if (threadIdx.x < nsc) hsc[threadIdx.x] = sc[threadIdx.x];
}
template <class T>
void cg_residual(long n, const double* al, const T* q, T* r, T* out, const T* sc, int nsc, T* hsc, T* partial,
                 cudaStream_t s) {
  launch_k(cg_residual_kernel<T>, dim3(md_grid(n)), dim3(TPB), 0, s, n, al, q, r,
           reinterpret_cast<unsigned char*>(partial), out, sc, nsc, hsc);
  COUNT_LAUNCH();
}

// The iterate: x += a p (CG), x2 = s (x2 + a p) and x += x2 (the smoothed form;
// its first iteration: x2 = s p, x = x2); with B also bt += al bp.  The first
// iteration's x and bt start from zero.
template <class T, bool SMOOTH, bool FIRST>
__global__ void __launch_bounds__(TPB) cg_iterate_kernel(long n, double a, double s, const T* __restrict__ p,
                                                         T* __restrict__ x2, T* __restrict__ x, double al,
                                                         const T* __restrict__ bp, T* __restrict__ bt) {
  pdl_begin();
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += (long)gridDim.x * TPB) {
    if (SMOOTH) {
      const T t = FIRST ? s * p[i] : s * axpy_re(a, p[i], x2[i]);
      x2[i] = t;
      x[i] = FIRST ? t : x[i] + t;
    } else {
      x[i] = axpy_re(a, p[i], FIRST ? T(0) : x[i]);
    }
    if (bt) bt[i] = axpy_re(al, bp[i], FIRST ? T(0) : bt[i]);
  }
}
template <class T>
void cg_iterate(long n, bool smooth, bool first, double a, double sc, const T* p, T* x2, T* x, double al, const T* bp, T* bt,
                cudaStream_t s) {
  auto go = [&](auto kern) { launch_k(kern, dim3(grid_1d(n)), dim3(TPB), 0, s, n, a, sc, p, x2, x, al, bp, bt); };
  if (smooth && first) go(cg_iterate_kernel<T, true, true>);
  else if (smooth) go(cg_iterate_kernel<T, true, false>);
  else if (first) go(cg_iterate_kernel<T, false, true>);
  else go(cg_iterate_kernel<T, false, false>);
  COUNT_LAUNCH();
}

// The Ritz vector and its residual: u = V y, r = W y + a bu (bu = u, or B y
// for the generalized problem), out[0] = r^H r (and out[1] = bu^H bu), y by
// value; one pass over the bases instead of one kernel per vector and one for
// the norm, with their roundings.
template <class T, bool GEP>
__global__ void __launch_bounds__(TPB) ritz_kernel(long n, int k, const T* __restrict__ V, const T* __restrict__ Wv,
                                                   const T* __restrict__ B, long ld, SmallVec<T> y, double a,
                                                   T* __restrict__ u, T* __restrict__ r, T* __restrict__ bu,
                                                   unsigned char* buf, T* out) {
  pdl_begin();
  T dot[GEP ? 2 : 1];
  dot[0] = T(0);
  if (GEP) dot[GEP] = T(0);
  const long step = (long)gridDim.x * TPB;
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += 2 * step) {  // two rows at once, as mdot
    const long at[2] = {i, i + step < n ? i + step : i};
    T su[2], sr[2], sb[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) su[q] = sr[q] = sb[q] = T(0);
#pragma unroll 2
    for (int c = 0; c < k; ++c)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        su[q] = fma_(V[at[q] + (long)c * ld], y.v[c], su[q]);
        sr[q] = fma_(Wv[at[q] + (long)c * ld], y.v[c], sr[q]);
        if (GEP) sb[q] = fma_(B[at[q] + (long)c * ld], y.v[c], sb[q]);
      }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (q == 1 && i + step >= n) break;
      T ub = su[q];
      u[at[q]] = ub;
      if (GEP) {
        ub = sb[q];
        bu[at[q]] = ub;
        dot[GEP] = fma_(cj(ub), ub, dot[GEP]);
      }
      const T t = axpy_re(a, ub, sr[q]);
      r[at[q]] = t;
      dot[0] = fma_(cj(t), t, dot[0]);
    }
  }
  md_finish<T, GEP ? 2 : 1>(dot, GEP ? 2 : 1, 0, buf, out);
}
template <class T>
void ritz(long n, int k, const T* V, const T* Wv, const T* B, long ld, const T* yh, double a, T* u, T* r, T* bu, T* out,
          T* partial, cudaStream_t s) {
  if (k < 1 || k > GMV_MAX) throw std::runtime_error("ritz: bad column count");
  SmallVec<T> y;
  for (int c = 0; c < k; ++c) y.v[c] = yh[c];
  auto go = [&](auto kern) {
    launch_k(kern, dim3(md_grid(n)), dim3(TPB), 0, s, n, k, V, Wv, B, ld, y, a, u, r, bu,
             reinterpret_cast<unsigned char*>(partial), out);
  };
  if (B) go(ritz_kernel<T, true>);
  else go(ritz_kernel<T, false>);
  COUNT_LAUNCH();
}

// Q (K x keep, leading dimension K, K <= 32) travels in the kernel's
// parameters: at most 16 KB for complex<double>, inside the 32 KB parameter
// space, so a restart needs no staging copy and no host synchronisation.
template <class T> struct SmallMat { T q[32 * 32]; };
template <class T>
__global__ void __launch_bounds__(TPB) rmult_kernel(long n, int K, int keep, const T* __restrict__ V, long ldv,
                                                    const __grid_constant__ SmallMat<T> Q, T* __restrict__ out) {
  pdl_begin();
  __shared__ T qs[32 * 32];
  for (int t = threadIdx.x; t < K * keep; t += TPB) qs[t] = Q.q[t];
  __syncthreads();
  for (long i = blockIdx.x * (long)TPB + threadIdx.x; i < n; i += (long)gridDim.x * TPB) {
    T row[32];
    for (int kk = 0; kk < K; ++kk) row[kk] = V[i + (long)kk * ldv];
    for (int c = 0; c < keep; ++c) {
      T acc = T(0);
      for (int kk = 0; kk < K; ++kk) acc = fma_(row[kk], qs[kk + c * K], acc);
      out[i + (long)c * n] = acc;
    }
  }
}
template <class T> void rmult(long n, int K, int keep, const T* V, long ldv, const T* Qh, T* out, cudaStream_t s) {
  if (K > 32 || keep > K) throw std::runtime_error("rmult: search space above 32");
  SmallMat<T> q;
  for (int c = 0; c < keep; ++c)
    for (int kk = 0; kk < K; ++kk) q.q[kk + c * K] = Qh[kk + c * K];
  launch_k(rmult_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, K, keep, V, ldv, q, out);
  COUNT_LAUNCH();
}

// ------------------------------------ the inner iteration in one launch ----
// The kernels above as the phases of one kernel.  Up to 1e5 rows a phase's bytes
// take well under a microsecond, and each kernel pays a launch and, most of
// them, a reduction tail (fence, atomic, partials read back: 3 us).  Here a
// phase ends in one barrier of the grid; its partial sums go to a buffer and
// every CTA adds them up itself in the order of md_finish, so there is no tail;
// the last reduction's partials go to pinned memory and are added by the host
// the same way.  A physical CTA holds VC of mdot's CTAs (256 threads each), so
// the order of every sum is that of the separate kernels.
// Bound: the chain of six phases, each a barrier, a few L2 latencies (0.14 us)
// and dependent float64 additions (some 50 cycles each), and from 1e5 rows on
// the FP64 units (2 FMA per SM and cycle).  us per iteration with 5 columns,
// separate kernels -> one (GB300): n = 4096 26.5 -> 20.5, 15625 29.8 -> 24.6,
// 64000 46.8 -> 26.7, 262144 59.3 -> 50.3, complex 262144 109 -> 102.
constexpr int kOneMaxCols = GMV_MAX;

// Grid barrier of a cooperative launch: the counter only grows, by gridDim.x
// per barrier, and `target` is its value once every CTA has arrived.  Gives up
// (false, in every thread) after `polls` polls.
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned target, int polls) {
  __shared__ bool ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    bool there = false;
    for (int t = 0; t < polls && !there; ++t) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
      there = (int)(v - target) >= 0;
    }
    ok = there;
  }
  __syncthreads();
  return ok;
}

template <class T> struct InnerOne {
  int n, g, k;                  // rows, md_grid(n), columns of the projection
  const T *U, *BU;              // N x k each, leading dimension n
  T *z, *r, *p;
  const int64_t *sptr, *bptr;   // A and, for GEP, B
  const int *col, *bcol;
  const T *val, *bval;
  double eta;                   // q = A p + eta (B) p
  bool first, posdef;
  T *rho, *hsc;
  const T* rho0;                // the previous iteration's rho (not read in the first)
  T* part;                      // (k + 3) g entries
  double* hpart;                // pinned, g entries: the partials of r^H r
  unsigned* bar;
  unsigned base;                // the barrier counter before this launch
  int polls;                    // after which a CTA gives up its wait, and leaves its partials unwritten
};

// x is written during the kernel: its loads stay out of the read-only path
template <class T>
__device__ __forceinline__ T sell_row(const SellBatch<T>& b, int64_t q, int64_t e, const int* __restrict__ col,
                                      const T* __restrict__ val, const T* x) {
  T w[kSellPre];
#pragma unroll
  for (int u = 0; u < kSellPre; ++u) w[u] = b.c[u] >= 0 ? x[b.c[u]] : T(0);
  T acc = T(0);
#pragma unroll
  for (int u = 0; u < kSellPre; ++u)
    if (b.c[u] >= 0) acc = fma_(b.v[u], w[u], acc);
  for (; q < e; q += 32) acc = fma_(val[q], x[__ldg(col + q)], acc);
  return acc;
}
constexpr int kOneRows = 2;  // rows of a thread (mdot's grid gives it that many from 4096 rows on)
// A thread keeps its rows of z, r, p and q in registers from
// phase to phase; p and r are the only vectors written (and B p for GEP, which
// the caller needs).  CLU: the grid is one thread-block cluster, whose barrier
// takes 0.75 us with the store before and the load after it; else a
// cooperative grid with grid_barrier (1.5 us).
template <class T, bool GEP, int VC, bool CLU>
__global__ void __launch_bounds__(TPB * VC, 1) inner_one_kernel(const __grid_constant__ InnerOne<T> a) {
  __shared__ T red[VC][MD_WARPS][MD_CH];
  __shared__ T ys[kOneMaxCols + 4 * VC];
  __shared__ double sc[2];
  const int vc = threadIdx.x / TPB, vt = threadIdx.x % TPB, vb = blockIdx.x * VC + vc;
  const int lane = threadIdx.x & 31, vw = vt >> 5;
  constexpr int RM = kOneRows;
  const bool on = vb < a.g;
  const int n = a.n, g = a.g, step = g * TPB, row0 = vb * TPB + vt;
  unsigned target = a.base;
  auto barrier = [&]() -> bool {
    if (CLU) {
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      return true;
    }
    return grid_barrier(a.bar, target += gridDim.x, a.polls);
  };
  auto has = [&](int j) { return on && row0 + j * step < n; };
  // the sums of the first nc columns over this virtual CTA's threads, as md_finish
  auto put = [&](auto& acc, int nc, auto* dst) {
    using E = std::remove_reference_t<decltype(acc[0])>;
    constexpr int CH = sizeof(acc) / sizeof(E);
    E* rd = reinterpret_cast<E*>(&red[vc][0][0]);
    const E v = md_tree(acc, lane);
    if (lane % (32 / CH) == 0) rd[vw * CH + md_col<CH>(lane)] = v;
    __syncthreads();
    if (vt < nc && on) {
      E t = E(0);
#pragma unroll
      for (int q = 0; q < MD_WARPS; ++q) t += rd[q * CH + vt];
      dst[(long)vt * g + vb] = t;
    }
    __syncthreads();
  };
  // sums over the grid of nc <= 4 columns' partials p, in md_finish's order, by this virtual CTA's warps; the caller
  // synchronises before it reads dst
  auto total = [&](const auto* p, int nc, auto* dst) {
    using E = std::remove_const_t<std::remove_reference_t<decltype(*p)>>;
    if (g <= 32) {
      if (vw < nc) {
        const E t = md_sum_32(p + (long)vw * g, g, lane);
        if (lane == 0) dst[vw] = t;
      }
      return;
    }
    E* rd = reinterpret_cast<E*>(&red[vc][0][0]);
    if (nc == 1) {
      E s[1];
      const E v = md_tree(*md_partials<E, 1>(p, nc, g, vw, lane, s), lane);
      if (lane == 0) rd[vw * 4] = v;
    } else if (nc > 0) {
      E s[4];
      const E v = md_tree(*md_partials<E, 4>(p, nc, g, vw, lane, s), lane);
      if (lane % 8 == 0) rd[vw * 4 + md_col<4>(lane)] = v;
    }
    __syncthreads();
    if (vt < nc) {
      E t = E(0);
#pragma unroll
      for (int q = 0; q < MD_WARPS; ++q) t += rd[q * 4 + vt];
      dst[vt] = t;
    }
  };
  T* pa = a.part;                                          // BU^H z
  double* pb = reinterpret_cast<double*>(pa + (long)a.k * g);  // Re r^H z
  T* pc = pa + (long)(a.k + 1) * g;                        // U^H q (and, for GEP, BU^H q)
  double* pd = pb;                                         // Re p^H q: pb is free again
  T z[RM], r[RM], p[RM], q[RM];
  // 1: the projection's coefficients
#pragma unroll
  for (int j = 0; j < RM; ++j) {
    z[j] = r[j] = p[j] = q[j] = T(0);
    if (has(j)) z[j] = a.z[row0 + j * step];
  }
  auto project = [&](auto ch, int c0) {
    constexpr int CH = decltype(ch)::value;
    const int nc = min(CH, a.k - c0);
    T acc[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) acc[c] = T(0);
#pragma unroll
    for (int j = 0; j < RM; ++j)
      if (has(j)) {
#pragma unroll
        for (int c = 0; c < CH; ++c)
          if (c < nc) acc[c] = fma_(cj(a.BU[row0 + j * step + (long)(c0 + c) * n]), z[j], acc[c]);
      }
    put(acc, nc, pa + (long)c0 * g);
  };
  for (int c0 = 0; c0 < a.k;) {  // a tree no wider than the columns left
    const int left = a.k - c0;
    if (left == 1) project(std::integral_constant<int, 1>(), c0++);
    else if (left <= 4 || sizeof(T) == 16) project(std::integral_constant<int, 4>(), c0), c0 += 4;
    else project(std::integral_constant<int, MD_CH>(), c0), c0 += MD_CH;
  }
#pragma unroll
  for (int j = 0; j < RM; ++j)
    if (has(j)) {
      r[j] = a.r[row0 + j * step];
      if (!a.first) p[j] = a.p[row0 + j * step];
    }
  if (!barrier()) return;
  // 2: z -= U c, rho = r^H z
  for (int c0 = 0; c0 < a.k; c0 += 4 * VC) {
    const int c = c0 + 4 * vc;
    total(pa + (long)c * g, min(4, max(0, a.k - c)), ys + c);
    __syncthreads();
  }
  {
    double dot[1] = {0.0};
    T acc[RM];
#pragma unroll
    for (int j = 0; j < RM; ++j) acc[j] = T(0);
#pragma unroll 4
    for (int c = 0; c < a.k; ++c) {
      const T y = ys[c];
#pragma unroll
      for (int j = 0; j < RM; ++j)
        if (has(j)) acc[j] = fma_(a.U[row0 + j * step + (long)c * n], y, acc[j]);
    }
#pragma unroll
    for (int j = 0; j < RM; ++j)
      if (has(j)) {
        z[j] = z[j] - acc[j];
        dot[0] = dot_re(r[j], z[j], dot[0]);
      }
    put(dot, 1, pb);
  }
  if (!barrier()) return;
  // 3: the search direction
  total((const double*)pb, vc == 0 ? 1 : 0, sc);
  if (threadIdx.x == 0) sc[1] = a.first ? 0.0 : sc[0] / rl(*a.rho0);
  __syncthreads();
  const double rho = sc[0];
  if (a.first) {
    if (!(rho == 0 || (a.posdef && rho <= 0)))
#pragma unroll
      for (int j = 0; j < RM; ++j)
        if (has(j)) a.p[row0 + j * step] = p[j] = z[j];
  } else {
    const double be = sc[1];
#pragma unroll
    for (int j = 0; j < RM; ++j)
      if (has(j)) a.p[row0 + j * step] = p[j] = axpy_re(be, p[j], z[j]);
  }
  // the rows' entries are loaded ahead of the barrier
  SellBatch<T> fa[RM];
  int64_t qa[RM], ea[RM];
#pragma unroll
  for (int j = 0; j < RM; ++j)
    if (has(j)) {
      const int i = row0 + j * step;
      qa[j] = a.sptr[i >> 5] + lane;
      ea[j] = a.sptr[(i >> 5) + 1];
      sell_load(fa[j], qa[j], ea[j], a.col, a.val);
    }
  if (!barrier()) return;
  // 4: q = A p + eta (B) p and its inner products
  {
    T dot[GEP ? 2 : 1];
    dot[0] = T(0);
    if (GEP) dot[GEP] = T(0);
#pragma unroll
    for (int j = 0; j < RM; ++j)
      if (has(j)) {
        const int i = row0 + j * step;
        const T acc = sell_row(fa[j], qa[j] + kSellPre * 32, ea[j], a.col, a.val, (const T*)a.p);
        T u = p[j];
        if (GEP) {
          const int64_t qb = a.bptr[i >> 5] + lane, eb = a.bptr[(i >> 5) + 1];
          SellBatch<T> fb;
          sell_load(fb, qb, eb, a.bcol, a.bval);
          u = sell_row(fb, qb + kSellPre * 32, eb, a.bcol, a.bval, (const T*)a.p);
          a.z[i] = u;
        }
        q[j] = axpy_re(a.eta, u, acc);
        dot[0] = fma_(cj(a.U[i]), q[j], dot[0]);
        if (GEP) dot[GEP] = fma_(cj(a.BU[i]), q[j], dot[GEP]);
      }
    put(dot, GEP ? 2 : 1, pc);
  }
  if (!barrier()) return;
  // 5: q -= BU (U^H q), p^H q
  total((const T*)pc, vc == 0 ? (GEP ? 2 : 1) : 0, ys);
  __syncthreads();
  const T uq = ys[0];
  {
    double dot[1] = {0.0};
#pragma unroll
    for (int j = 0; j < RM; ++j)
      if (has(j)) {
        q[j] = q[j] - fma_(a.BU[row0 + j * step], uq, T(0));
        dot[0] = dot_re(p[j], q[j], dot[0]);
      }
    put(dot, 1, pd);
  }
  if (!barrier()) return;
  // 6: r -= (rho / p^H q) q, r^H r
  total((const double*)pd, vc == 0 ? 1 : 0, sc);
  if (threadIdx.x == 0) sc[1] = -1.0 * (rho / sc[0]);
  __syncthreads();
  const double al = sc[1];
  double dot[1] = {0.0};
#pragma unroll
  for (int j = 0; j < RM; ++j)
    if (has(j)) {
      r[j] = axpy_re(al, q[j], r[j]);
      a.r[row0 + j * step] = r[j];
      dot[0] = dot_re(r[j], r[j], dot[0]);
    }
  put(dot, 1, a.hpart);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *a.rho = T(rho);
    a.hsc[0] = T(rho);
    a.hsc[1] = uq;
    a.hsc[2] = GEP ? ys[1] : T(0);
    a.hsc[3] = T(sc[0]);
  }
}

// md_finish's order on the host, for real partial sums
double md_sum_host(const double* p, int g) {
  if (g == 1) return p[0];
  double t = 0;
  for (int w = 0; w < MD_WARPS && 32 * w < g; ++w) {
    double s[32];
    for (int l = 0; l < 32; ++l) {
      s[l] = 0;
      for (int q = 32 * w + l; q < g; q += TPB) s[l] += p[q];
    }
    for (int o = 16; o > 0; o >>= 1)
      for (int l = 0; l < o; ++l) s[l] += s[l + o];
    t += s[0];
  }
  return t;
}

// The launch shapes of inner_one_kernel and, per device, the most (virtual)
// CTAs each runs at once: the hardware's answer, not an assumption about it.
enum { kOneCluster, kOneGrid, kOneGrid4, kOneShapes };
template <class T> struct OneShape {
  void (*kern)(InnerOne<T>);
  int vc;
  bool clu;
};
template <class T> static OneShape<T> one_shape(int shape, bool gep) {
  switch (shape) {
    case kOneCluster: return {gep ? inner_one_kernel<T, true, 1, true> : inner_one_kernel<T, false, 1, true>, 1, true};
    case kOneGrid: return {gep ? inner_one_kernel<T, true, 1, false> : inner_one_kernel<T, false, 1, false>, 1, false};
    default: return {gep ? inner_one_kernel<T, true, 4, false> : inner_one_kernel<T, false, 4, false>, 4, false};
  }
}
static void one_cluster(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int g) {
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = g;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}
template <class T> static int one_most(int shape, bool gep) {
  static std::mutex mu;
  static std::map<int, int> most;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  const int key = (dev * kOneShapes + shape) * 2 + gep;
  auto it = most.find(key);
  if (it != most.end()) return it->second;
  const OneShape<T> o = one_shape<T>(shape, gep);
  int m = 0;
  if (o.clu) {
    for (int g : {16, 8}) {
      if (m) break;
      if (g > 8 && cudaFuncSetAttribute(o.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        continue;
      }
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      cfg.gridDim = dim3(g);
      cfg.blockDim = dim3(TPB);
      one_cluster(cfg, at, g);
      int nc = 0;
      if (cudaOccupancyMaxActiveClusters(&nc, o.kern, &cfg) == cudaSuccess && nc > 0) m = g;
      else cudaGetLastError();
    }
  } else {
    int per = 0, sms = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, o.kern, TPB * o.vc, 0));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    m = per > 0 ? sms * o.vc : 0;
  }
  return most[key] = m;
}
// Which shape, if any.  Two rows per thread fit in registers: mdot's grid has
// that many from 4096 rows on, up to its cap of 1216 CTAs.  Below, it has one
// or two CTAs, whose one or two SMs then bound every phase (n = 1000: 30.7 us
// in one launch, 23.6 us in seven kernels whose product and update spread over
// the grid).  Up to 16 CTAs (n = 8192) one cluster, whose barrier is the
// cheapest; then one CTA per SM (n = 77824), then four of mdot's CTAs in each
// (n = 311296); beyond, the separate kernels.
template <class T> static int one_pick(long n, bool gep) {
  const int g = md_grid(n);
  const int rows = (int)((n + (long)g * TPB - 1) / ((long)g * TPB));
  if (rows > kOneRows) return -1;
  for (int shape : {kOneCluster, kOneGrid, kOneGrid4})
    if (g <= one_most<T>(shape, gep)) return shape;
  return -1;
}
template <class T> bool inner_one_ok(long n, int k, bool gep) { return k <= kOneMaxCols && one_pick<T>(n, gep) >= 0; }
template <class T>
int inner_one(const SellMatrix<T>& A, const SellMatrix<T>* B, int k, const T* U, const T* BU, T* z, T* r, T* p, double eta,
              bool first, bool posdef, T* rho, const T* rho0, T* hsc, T* part, double* hpart, unsigned* bar, OneState& st,
              cudaStream_t s) {
  InnerOne<T> a;
  a.n = A.n;
  a.g = md_grid(A.n);
  a.k = k;
  a.U = U;
  a.BU = BU;
  a.z = z;
  a.r = r;
  a.p = p;
  a.sptr = A.sptr;
  a.col = A.col;
  a.val = A.val;
  a.bptr = B ? B->sptr : nullptr;
  a.bcol = B ? B->col : nullptr;
  a.bval = B ? B->val : nullptr;
  a.eta = eta;
  a.first = first;
  a.posdef = posdef;
  a.rho = rho;
  a.rho0 = rho0;
  a.hsc = hsc;
  a.part = part;
  a.hpart = hpart;
  a.bar = bar;
  a.base = st.base;
  a.polls = st.polls;
  const OneShape<T> o = one_shape<T>(one_pick<T>(A.n, B != nullptr), B != nullptr);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.g + o.vc - 1) / o.vc);
  cfg.blockDim = dim3(TPB * o.vc);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  if (o.clu) {
    one_cluster(cfg, at, a.g);
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
  }
  CK(cudaLaunchKernelEx(&cfg, o.kern, a));
  if (!o.clu) st.base += 5u * cfg.gridDim.x;
  COUNT_LAUNCH();
  return a.g;
}

template <class T> __global__ void diag_kernel(long n, const double* __restrict__ d, const T* __restrict__ r, T* x) {
  pdl_begin();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    x[i] = d[i] * r[i];
}
template <class T> void diagsolve(long n, const double* d, const T* rhs, T* sol, cudaStream_t s) {
  launch_k(diag_kernel<T>, dim3(grid_1d(n)), dim3(TPB), 0, s, n, d, rhs, sol);
  COUNT_LAUNCH();
}

// ------------------------------------------------ multilevel LDL^H apply ----
// Entries q, q + step, ... (below e) of a row, U at a time: a batch's
// column indices and values are loaded together, then its gathers of y, and
// the products are added in entry order, so the roundings are those of one
// entry at a time while U dependent load chains are in flight.  kUnr for the
// sweeps; the external-entry gathers of large dense blocks (rows of hundreds
// of entries) take kUnrLong.
constexpr int kUnr = 4;
constexpr int kUnrLong = 8;
template <class A, int U> struct EntBatch {
  int c[U];
  A v[U];
};
template <bool NC, class A, int U, class S>
__device__ __forceinline__ void ent_load(EntBatch<A, U>& b, int64_t q, int64_t e, int step, const int* __restrict__ ci,
                                         const S* __restrict__ cv) {
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t qq = q + (int64_t)u * step;
    if (qq < e) {
      b.c[u] = NC ? ld_idx_nc(ci + qq) : ci[qq];
      b.v[u] = NC ? ldan<A>(cv + qq) : lda<A>(cv + qq);
    } else {
      b.c[u] = -1;
      b.v[u] = A(0);
    }
  }
}
// nu: how many entries of the batch any lane of the warp may have (a bound that
// is the same in all lanes lets the warp skip the rest).
template <class A, int U>
__device__ __forceinline__ A ent_use(const EntBatch<A, U>& b, const A* y, A acc, int nu = U) {
  A w[U];
#pragma unroll
  for (int u = 0; u < U; ++u) w[u] = u < nu && b.c[u] >= 0 ? y[b.c[u]] : A(0);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u < nu && b.c[u] >= 0) acc = fma_(b.v[u], w[u], acc);
  return acc;
}
// The longest of a warp's rows, and the tree over the LANES lanes of a row
// whose sums lie in its first lanes: steps that would only add zeros (rows of
// at most o entries leave the lanes from o on empty) are left out.  Short rows
// are the rule in the first and last levels, and a float64 addition occupies
// the SM's FP64 unit for 16 cycles per warp whether its lanes are zero or not.
// us per application (GB300): tridiagonal n = 1000 28.7 -> 22.6, FEM 384^2 291
// -> 276, Anderson 56^3 350 -> 339, 40^3 151 -> 149, Laplacian 20^3 58.2 -> 56.7.
// Lengths are exact up to kLongest, which no caller reaches: batch counts
// derived from a smaller cap would drop the entries beyond it.
constexpr int kLongest = 1 << 30;
__device__ __forceinline__ int warp_longest(int64_t len) {
  return __reduce_max_sync(0xffffffffu, (int)(len < 0 ? 0 : len < kLongest ? len : kLongest));
}
template <int LANES, class A> __device__ __forceinline__ A row_sum(A v, int longest) {
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1)
    if (o < longest) v = v + shfl_xor_any(v, o);
  return v;
}
// entries [q, e) of a row beyond its first batch, into L2 ahead of use
template <class S>
__device__ __forceinline__ void prefetch_rest(int64_t q, int64_t e, const int* __restrict__ ci,
                                              const S* __restrict__ cv) {
  if (q < e) {
    l2_prefetch(ci + q, sizeof(int) * (size_t)(e - q));
    l2_prefetch(cv + q, sizeof(S) * (size_t)(e - q));
  }
}
// The batches of a row in a pipeline of one: the next batch's entries are
// loaded before the current one's gathers are waited for.
template <bool NC, int U = kUnr, class A, class S>
__device__ __forceinline__ A ent_dot(int64_t q, int64_t e, int step, const int* __restrict__ ci,
                                     const S* __restrict__ cv, const A* y, A acc) {
  if (q < e) {
    EntBatch<A, U> b;
    ent_load<NC>(b, q, e, step, ci, cv);
    for (;;) {
      q += (int64_t)U * step;
      if (q >= e) return ent_use(b, y, acc);
      EntBatch<A, U> nx;
      ent_load<NC>(nx, q, e, step, ci, cv);
      acc = ent_use(b, y, acc);
      b = nx;
    }
  }
  return acc;
}
// The same for a kernel that loaded its first two batches before its wait for
// y.  Measured (GB300, us per application, without -> with): Anderson 56^3
// float32 377 -> 364, Laplacian 20^3 69.1 -> 65.8, tight-binding 48^3 166.2 ->
// 163.5, FEM 384^2 302 -> 299; batches of eight instead: 362, 70.7, 184, 339.
template <bool NC, int U, class A, class S>
__device__ __forceinline__ A ent_pipe(EntBatch<A, U>& b, int64_t q, int64_t e, int step, const int* __restrict__ ci,
                                      const S* __restrict__ cv, EntBatch<A, U>& nx, const A* y, int nu) {
  A acc = A(0);
  q += (int64_t)U * step;  // nx holds the batch at q when q < e
  if (nu < U) return ent_use(b, y, acc, nu);
  while (q < e) {
    acc = ent_use(b, y, acc);
    b = nx;
    q += (int64_t)U * step;
    if (q < e) ent_load<NC>(nx, q, e, step, ci, cv);
  }
  return ent_use(b, y, acc);
}

template <class T, class A>
__global__ void ildl_gather_kernel(int n, const int* __restrict__ orig, const T* __restrict__ b, A* __restrict__ y) {
  pdl_launch();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int o = orig[s];
  pdl_wait();
  y[s] = cvt<A>(b[o]);
}
template <class T, class A>
__global__ void ildl_scatter_kernel(int n, const int* __restrict__ orig, const A* __restrict__ y, T* __restrict__ x) {
  pdl_launch();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int o = orig[s];
  pdl_wait();
  x[o] = cvt<T>(y[s]);
}
template <class S, class A>
__global__ void ildl_dsolve_kernel(int n, const signed char* __restrict__ blk, const int* __restrict__ partner,
                                   const S* __restrict__ dv, const S* __restrict__ dof, A* __restrict__ y) {
  pdl_launch();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  signed char b = blk[s];
  if (b == 1) {
    const A d = lda<A>(dv + s);
    pdl_wait();
    y[s] = d * y[s];
  } else if (b == 2) {
    const int t = partner[s];
    const A o = lda<A>(dof + s), d0 = lda<A>(dv + s), d1 = lda<A>(dv + t);
    pdl_wait();
    A a0 = y[s], a1 = y[t];
    y[s] = fma_(d0, a0, o * a1);
    y[t] = fma_(cj(o), a0, d1 * a1);
  }
}
// A run of narrow levels [l0, l1) in one CTA: a warp per row, levels
// separated by __syncthreads (which orders the CTA's global writes).
__device__ __forceinline__ float wsum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double wsum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ cc wsum(cc v) { return cc(wsum(v.x), wsum(v.y)); }
__device__ __forceinline__ zc wsum(zc v) { return zc(wsum(v.x), wsum(v.y)); }

constexpr int RUN_TPB = 1024;
constexpr int RUN_WARPS = RUN_TPB / 32;
// A level with R < 32 rows gives each row 32/R warps; their partial sums are
// added in a fixed order after a barrier, so results do not depend on timing.
// Bound for float64: the one SM's FP64 unit, which is why sums over empty lanes
// and warps are left out (row_sum).
template <class S, class A>
__global__ void __launch_bounds__(RUN_TPB) ildl_run_kernel(int l0, int l1, const int* __restrict__ lptr,
                                                          const int* __restrict__ rows, const int64_t* __restrict__ rp,
                                                          const int* __restrict__ ci, const S* __restrict__ cv,
                                                          A* y) {
  pdl_begin();
  __shared__ A part[RUN_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int l = l0; l < l1; ++l) {
    const int lo = lptr[l], hi = lptr[l + 1], R = hi - lo;
    // the sum of this warp's entries of row s: from entry `off` of the row on, every `step`
    auto sum = [&](int s, int off, int step) {
      const int64_t b = rp[s], e = rp[s + 1];
      const int len = warp_longest(e - b - off), nu = (len + step - 1) / step;
      A acc;
      if (nu <= kUnr) {
        EntBatch<A, kUnr> first;
        ent_load<false>(first, b + off + lane, e, step, ci, cv);
        acc = ent_use(first, (const A*)y, A(0), nu);
      } else {
        acc = ent_dot<false>(b + off + lane, e, step, ci, cv, (const A*)y, A(0));
      }
      return row_sum<32>(acc, len);
    };
    if (R >= RUN_WARPS) {
      for (int t = lo + warp; t < hi; t += RUN_WARPS) {
        const int s = rows ? rows[t] : t;
        const A own = y[s];
        const A acc = sum(s, 0, 32);
        if (lane == 0) y[s] = own - acc;
      }
      __syncthreads();
    } else {
      int G = RUN_WARPS / R;
      G = 1 << (31 - __clz(G));
      const int slot = warp / G, sub = warp % G;
      int s = -1, parts = 0;  // the row and how many of its G warps have entries
      A own = A(0);
      if (slot < R) {
        s = rows ? rows[lo + slot] : lo + slot;
        own = y[s];
        parts = (warp_longest(rp[s + 1] - rp[s]) + 31) / 32;
        parts = parts < G ? parts : G;
        const A acc = sub < parts ? sum(s, sub * 32, 32 * G) : A(0);
        if (lane == 0) part[warp] = acc;
      }
      __syncthreads();
      if (slot < R && sub == 0 && lane == 0) {
        A t = part[warp];
        for (int j = 1; j < parts; ++j) t = t + part[warp + j];
        y[s] = own - t;
      }
      __syncthreads();
    }
  }
}
// One wide level: LANES lanes per row (8, 16 or 32, from the level's mean
// row length, so long rows are read by more lanes at once).
//
// Blocks of 128 threads free their SM slots in smaller pieces than 256 did, and
// a float64 level lets its successor start only once it has its own y (kLate):
// the successor's blocks, there to load their entries, otherwise take turns on
// the FP64 units and slots this level still needs.  us per application (GB300),
// 256 threads and early -> as here: FEM 384^2 float64 276 -> 238, tight-binding
// 48^3 complex128 386 -> 277, Anderson 44^3 float64 361 -> 340; float32, were it
// late as well: FEM 127.6 -> 131.5, Anderson 44^3 155.6 -> 156.8.  A float64 tile
// product (tri_cluster_kernel) lets it start once its products are done: FEM
// 384^2 239 -> 232, a FEM 512^2 solve 214.5 -> 211.1 ms.
constexpr int WIDE_TPB = 128;
template <class A> constexpr bool kLate = sizeof(A) == 16 || std::is_same<A, double>::value;
static inline int lanes_for(double entries_per_row) {
  return entries_per_row >= 48 ? 32 : entries_per_row >= 20 ? 16 : 8;
}
int lanes_per_row(double entries_per_row) { return lanes_for(entries_per_row); }
template <class S, class A, int LANES>
__global__ void __launch_bounds__(WIDE_TPB) ildl_wide_kernel(int lo, int hi, const int* __restrict__ rows,
                                                            const int64_t* __restrict__ rp, const int* __restrict__ ci,
                                                            const S* __restrict__ cv, A* __restrict__ y) {
  if (!kLate<A>) pdl_launch();
  const int g = blockIdx.x * (WIDE_TPB / LANES) + (threadIdx.x / LANES);
  const int lane = threadIdx.x % LANES;
  const int t = lo + g;
  const bool ok = t < hi;
  int s = 0;
  int64_t b = 0, e = 0;
  if (ok) {
    s = rows ? rows[t] : t;
    b = rp[s] + lane;
    e = rp[s + 1];
    if (lane == 0) prefetch_rest(b + kUnr * LANES, e, ci, cv);
  }
  EntBatch<A, kUnr> first, second;
  const int longest = warp_longest(ok ? e - b + lane : 0);
  ent_load<false>(first, b, e, LANES, ci, cv);
  ent_load<false>(second, b + kUnr * LANES, e, LANES, ci, cv);
  pdl_wait();
  if (kLate<A>) pdl_launch();
  const A own = ok && lane == 0 ? y[s] : A(0);  // requested with the gathers, not after the sum
  A acc = ent_pipe<false, kUnr>(first, b, e, LANES, ci, cv, second, (const A*)y, (longest + LANES - 1) / LANES);
  acc = row_sum<LANES>(acc, longest);
  if (ok && lane == 0) y[s] = own - acc;
}

// Rows [s0, s0 + m) of a block: y[s0 + t] -= sum of row t's entries (local
// row pointers, global columns), LANES lanes per row.
// out[t] = y[s0 + t] - sum of row t's entries (out may be y + s0).  NC: the
// entries and column indices are read without L1 allocation, which keeps L1
// for the gathered y; measured on GB300 it pays for blocks with a million or
// more external entries (Anderson 50^3 application 0.387 -> 0.356 ms with it
// on every block) and costs a little on smaller ones (40^3: 0.198 -> 0.202).
template <class S, class A, int LANES, bool NC>
__global__ void __launch_bounds__(WIDE_TPB) tail_ext_kernel(int m, int s_tail, const int64_t* __restrict__ rp,
                                                           const int* __restrict__ ci, const S* __restrict__ cv,
                                                           const A* y, A* out) {
  pdl_launch();
  constexpr int U = NC ? kUnrLong : kUnr;
  const int t = blockIdx.x * (WIDE_TPB / LANES) + (threadIdx.x / LANES);
  const int lane = threadIdx.x % LANES;
  int64_t b = 0, e = 0;
  if (t < m) {
    b = rp[t] + lane;
    e = rp[t + 1];
    if (lane == 0) prefetch_rest(b + U * LANES, e, ci, cv);
  }
  EntBatch<A, U> first, second;
  const int longest = warp_longest(t < m ? e - b + lane : 0);
  ent_load<NC>(first, b, e, LANES, ci, cv);
  ent_load<NC>(second, b + U * LANES, e, LANES, ci, cv);
  pdl_wait();
  const A own = t < m && lane == 0 ? y[s_tail + t] : A(0);
  A acc = ent_pipe<NC, U>(first, b, e, LANES, ci, cv, second, y, (longest + LANES - 1) / LANES);
  acc = row_sum<LANES>(acc, longest);
  if (t < m && lane == 0) out[t] = own - acc;
}
template <class S, class A>
static void launch_wide(int lanes, int lo, int hi, const int* rows, const int64_t* rp, const int* ci, const S* cv, A* y,
                        cudaStream_t s) {
  const int nb = (hi - lo) * lanes / WIDE_TPB + 1;
  if (lanes == 32) launch_k(ildl_wide_kernel<S, A, 32>, dim3(nb), dim3(WIDE_TPB), 0, s, lo, hi, rows, rp, ci, cv, y);
  else if (lanes == 16) launch_k(ildl_wide_kernel<S, A, 16>, dim3(nb), dim3(WIDE_TPB), 0, s, lo, hi, rows, rp, ci, cv, y);
  else launch_k(ildl_wide_kernel<S, A, 8>, dim3(nb), dim3(WIDE_TPB), 0, s, lo, hi, rows, rp, ci, cv, y);
}
constexpr int64_t kExtStreamEntries = 1 << 20;  // external entries from which tail_ext streams them
template <class S, class A, bool NC>
static void launch_ext_(int lanes, int m, int s0, const int64_t* rp, const int* ci, const S* cv, const A* y, A* out,
                        cudaStream_t s) {
  const int nb = m * lanes / WIDE_TPB + 1;
  if (lanes == 32) launch_k(tail_ext_kernel<S, A, 32, NC>, dim3(nb), dim3(WIDE_TPB), 0, s, m, s0, rp, ci, cv, y, out);
  else if (lanes == 16) launch_k(tail_ext_kernel<S, A, 16, NC>, dim3(nb), dim3(WIDE_TPB), 0, s, m, s0, rp, ci, cv, y, out);
  else launch_k(tail_ext_kernel<S, A, 8, NC>, dim3(nb), dim3(WIDE_TPB), 0, s, m, s0, rp, ci, cv, y, out);
}
template <class S, class A>
static void launch_ext(int lanes, int m, int s0, const int64_t* rp, const int* ci, const S* cv, A* y, A* out,
                       int64_t entries, cudaStream_t s) {
  if (entries >= kExtStreamEntries) launch_ext_<S, A, true>(lanes, m, s0, rp, ci, cv, y, out, s);
  else launch_ext_<S, A, false>(lanes, m, s0, rp, ci, cv, y, out, s);
}
// The sequential part of a tail sweep in one CTA.  Shared memory holds the
// tail of y (yt), the row pointers relative to the first tail entry, the level
// pointers and (backward sweep) the row order, so a level costs one global
// load of entries, which is issued for the next level before the barrier.
// Rows of small levels are split over several warps as in ildl_run_kernel.
template <class A> __host__ __device__ constexpr size_t tail_smem_bytes(int m, int nlev, bool rows) {
  return ((sizeof(A) * (size_t)m + 15) / 16) * 16 + 4 * (size_t)(m + 1) + 4 * (size_t)(nlev + 1) +
         (rows ? 4 * (size_t)m : 0);
}
template <class S, class A>
__global__ void __launch_bounds__(RUN_TPB) tail_run_kernel(int m, int s_tail, int nlev, const int* __restrict__ lptr,
                                                          const int* __restrict__ rows, const int64_t* __restrict__ rp,
                                                          const int* __restrict__ ci, const S* __restrict__ cv,
                                                          A* __restrict__ y) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A* yt = reinterpret_cast<A*>(smem_raw);
  int* srp = reinterpret_cast<int*>(smem_raw + ((sizeof(A) * (size_t)m + 15) / 16) * 16);
  int* slp = srp + (m + 1);
  int* srw = slp + (nlev + 1);
  __shared__ A part[RUN_WARPS];
  const int64_t base = rp[0];
  for (int t = threadIdx.x; t < m; t += RUN_TPB) {
    yt[t] = y[s_tail + t];
    if (rows) srw[t] = rows[t];
  }
  for (int t = threadIdx.x; t <= m; t += RUN_TPB) srp[t] = (int)(rp[t] - base);
  for (int t = threadIdx.x; t <= nlev; t += RUN_TPB) slp[t] = lptr[t];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // this warp's row r, entry range [q0, q1) with stride `step` in level l
  auto assign = [&](int l, int& r, int& q0, int& q1, int& step, int& G, int& slot, int& sub) {
    const int lo = slp[l], R = slp[l + 1] - lo;
    if (R >= RUN_WARPS) {
      G = 1;
      slot = warp;
      sub = 0;
    } else {
      G = RUN_WARPS / R;
      G = 1 << (31 - __clz(G));
      slot = warp / G;
      sub = warp % G;
    }
    step = 32 * G;
    if (slot < R) {
      const int t = lo + slot;
      r = rows ? srw[t] : t;
      q0 = srp[r] + sub * 32 + lane;
      q1 = srp[r + 1];
    } else {
      r = -1;
      q0 = q1 = 0;
    }
  };
  int r = -1, q0 = 0, q1 = 0, step = 32, G = 1, slot = 0, sub = 0;
  int pci = 0;
  A pcv = A(0);
  if (nlev > 0) {
    assign(0, r, q0, q1, step, G, slot, sub);
    if (q0 < q1) {
      pci = ci[base + q0];
      pcv = lda<A>(cv + base + q0);
    }
  }
  for (int l = 0; l < nlev; ++l) {
    const int lo = slp[l], hi = slp[l + 1], R = hi - lo;
    A acc = A(0);
    if (q0 < q1) {
      acc = pcv * yt[pci];
      for (int q = q0 + step; q < q1; q += step) acc = fma_(lda<A>(cv + base + q), yt[ci[base + q]], acc);
    }
    acc = wsum(acc);
    if (R >= RUN_WARPS) {
      if (lane == 0 && r >= 0) yt[r] = yt[r] - acc;
      for (int t = lo + warp + RUN_WARPS; t < hi; t += RUN_WARPS) {  // further rows of this warp
        const int rr = rows ? srw[t] : t;
        A a2 = A(0);
        for (int q = srp[rr] + lane; q < srp[rr + 1]; q += 32) a2 = fma_(lda<A>(cv + base + q), yt[ci[base + q]], a2);
        a2 = wsum(a2);
        if (lane == 0) yt[rr] = yt[rr] - a2;
      }
    } else if (lane == 0) {
      part[warp] = acc;
    }
    int nr = -1, nq0 = 0, nq1 = 0, nstep = 32, nG = 1, nslot = 0, nsub = 0;
    if (l + 1 < nlev) {  // prefetch the first entry of the next level
      assign(l + 1, nr, nq0, nq1, nstep, nG, nslot, nsub);
      if (nq0 < nq1) {
        pci = ci[base + nq0];
        pcv = lda<A>(cv + base + nq0);
      }
    }
    __syncthreads();
    if (R < RUN_WARPS) {
      if (slot < R && sub == 0 && lane == 0) {
        A t = part[warp];
        for (int j = 1; j < G; ++j) t = t + part[warp + j];
        yt[r] = yt[r] - t;
      }
      __syncthreads();
    }
    r = nr; q0 = nq0; q1 = nq1; step = nstep; G = nG; slot = nslot; sub = nsub;
  }
  for (int t = threadIdx.x; t < m; t += RUN_TPB) y[s_tail + t] = yt[t];
}

constexpr int TRI_TPB = 256;  // threads per CTA of the tile kernel
constexpr int kTriDepth = 3;  // units of its chunk that a thread has in flight

// 16-byte read-only load of data read once per launch (tiles): issued as
// written, kept in its registers (no re-load at the point of use), no L1 allocation
__device__ __forceinline__ uint4 ld_stream(const uint4* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}

// Dense block product y = T x over a set of 64 x 64 tiles (column-major
// inside a tile), with the reduction inside a thread-block cluster: the CL
// CTAs of a cluster (8, or 16 where the GPU allows that non-portable size)
// share one tile row and each streams a contiguous chunk of its tiles
// (16-byte vectors of V consecutive rows of one tile column per thread;
// per-column partial sums added in a fixed order).  Each CTA puts its
// 64-vector into rank 0's shared memory; rank 0 adds the CL vectors in rank
// order and writes the row, so results do not depend on timing.  x must not
// alias y.  The cluster size is a launch attribute (launch_tri), never left to
// a default.
//
// Bound: the tiles' bytes, for float64 also the FP64 units (2 FMA per SM and
// cycle), and the chain of tiles of the longest row, ceil(row / CL).  So a
// thread keeps kTriDepth units of up to four vectors (and their x) in flight,
// the first ones before it waits for x; the longest rows start first (rev: the
// longest is the last row); and nothing is requested into L2 ahead.  us per
// application (GB300), one tile at a time with the rest of the chunk
// prefetched into L2 -> now: Laplacian 20^3 float64 72.2 -> 69.0, Anderson
// 28^3 float64 205.7 -> 166.6, float32 70.3 -> 67.5, 40^3 186.6 -> 162.1, 56^3
// 431 -> 375, 25^3 bfloat16 46.1 -> 47.3.
template <class S, class A, int CL>
__global__ void __launch_bounds__(TRI_TPB)
    tri_cluster_kernel(const int4* __restrict__ items, bool rev, const S* __restrict__ tiles, const A* __restrict__ x,
                       int m, A* __restrict__ y) {
  if (!kLate<A>) pdl_launch();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr int V = 16 / sizeof(S);
  constexpr int RG = 64 / V;
  constexpr int CPS = TRI_TPB / RG;
  constexpr int NS = 64 / CPS;
  constexpr int DEPTH = kTriDepth;
  constexpr int UN = NS < 4 ? NS : 4;   // vectors per unit
  constexpr int PER = NS / UN;          // units per tile
  __shared__ A red[CPS][64];
  __shared__ A part[CL][64];
  const int cid = blockIdx.x / CL, ncl = gridDim.x / CL;
  const int4 it = items[(rev ? ncl - 1 - cid : cid) * CL + blockIdx.x % CL];
  const int nu = it.z * PER;
  const int rg = threadIdx.x % RG, cs = threadIdx.x / RG;
  A acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = A(0);
  const uint4* tp = reinterpret_cast<const uint4*>(tiles) + (size_t)it.y * (64 * 64 / V) + threadIdx.x;
  const int c0 = it.w * 64 + cs;
  auto load = [&](int u, uint4* buf) {
#pragma unroll
    for (int sl = 0; sl < UN; ++sl) buf[sl] = ld_stream(tp + ((size_t)u * UN + sl) * TRI_TPB);
  };
  auto xload = [&](int u, A* xv) {
#pragma unroll
    for (int sl = 0; sl < UN; ++sl) {
      const int c = c0 + (u * UN + sl) * CPS;
      xv[sl] = c < m ? x[c] : A(0);
    }
  };
  uint4 buf[DEPTH][UN];
  A xv[DEPTH][UN];
#pragma unroll
  for (int d = 0; d < DEPTH; ++d)
    if (d < nu) load(d, buf[d]);
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  pdl_wait();
#pragma unroll
  for (int d = 0; d < DEPTH; ++d)
    if (d < nu) xload(d, xv[d]);
  for (int u0 = 0; u0 < nu; u0 += DEPTH) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      const int u = u0 + d;
      if (u < nu) {
#pragma unroll
        for (int sl = 0; sl < UN; ++sl) {
          const S* e = reinterpret_cast<const S*>(&buf[d][sl]);
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v] = fma_(lda<A>(e + v), xv[d][sl], acc[v]);
        }
        if (u + DEPTH < nu) {
          load(u + DEPTH, buf[d]);
          xload(u + DEPTH, xv[d]);
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < V; ++v) red[cs][V * rg + v] = acc[v];
  __syncthreads();
  A sum = A(0);
  if (threadIdx.x < 64) {
    sum = red[0][threadIdx.x];
#pragma unroll
    for (int j = 1; j < CPS; ++j) sum = sum + red[j][threadIdx.x];
  }
  if (kLate<A>) pdl_launch();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x < 64) *cl.map_shared_rank(&part[cl.block_rank()][threadIdx.x], 0) = sum;
  cl.sync();
  if (cl.block_rank() == 0 && threadIdx.x < 64) {
    A t = A(0);
#pragma unroll
    for (int r = 0; r < CL; ++r) t = t + part[r][threadIdx.x];
    const int e = it.x * 64 + threadIdx.x;
    if (e < m) y[e] = t;
  }
}

// one launch of a cluster kernel: cl CTAs per cluster, PDL as launch_k
template <class... Params, class... Args>
static void launch_cl(void (*kern)(Params...), dim3 grid, dim3 block, int cl, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = g_pdl ? 2 : 1;
  CK(cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...));
}
// items are grid-sized multiples of the cluster size (make_cluster_items)
template <class S, class A>
static void launch_tri(int items, int cl, bool lower, const int4* it, const S* tiles, const A* x, int m, A* y, cudaStream_t s) {
  if (cl == 16) launch_cl(tri_cluster_kernel<S, A, 16>, dim3(items), dim3(TRI_TPB), 16, s, it, lower, tiles, x, m, y);
  else launch_cl(tri_cluster_kernel<S, A, 8>, dim3(items), dim3(TRI_TPB), 8, s, it, lower, tiles, x, m, y);
}
// Whether clusters of 16 tile CTAs can run on the current device: allows the
// non-portable size on both instantiations' kernel and asks the occupancy
// calculator for at least one active cluster.  Called on upload, before any
// graph capture.
template <class S, class A> bool tri_cluster16_ok() {
  auto kern = tri_cluster_kernel<S, A, 16>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16);
  cfg.blockDim = dim3(TRI_TPB);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int nc = 0;
  if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return nc > 0;
}

// raise the dynamic shared-memory limit of the tail kernel once per size
// (done before any graph capture: ildl_apply_graph calls it first)
template <class S, class A> static void ensure_tail_smem(size_t bytes) {
  // the attribute applies to the current device only: one raised size per device
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static size_t set[kMaxDev] = {};
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  size_t& cur = set[dev < kMaxDev ? dev : kMaxDev - 1];
  if (dev >= kMaxDev || bytes > std::max<size_t>(cur, 48 * 1024)) {
    CK(cudaFuncSetAttribute(tail_run_kernel<S, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    cur = std::max(cur, bytes);
  }
}

constexpr int kRunRows = 2 * RUN_WARPS;
constexpr int64_t kRunEntries = 16384;
template <class S>
void ildl_plan(DevFactor<S>& F, const std::vector<int64_t>& lp, const std::vector<int64_t>& up,
               const std::vector<int>& brows) {
  auto plan = [&](const std::vector<int>& ptr, bool fwd, std::vector<int>& seg) {
    seg.clear();
    const int nl = (int)ptr.size() - 1;
    int l = 1;  // level 0 has no off-diagonal entries in either sweep
    while (l < nl) {
      auto work = [&](int lv) {
        int64_t nz = 0;
        for (int t = ptr[lv]; t < ptr[lv + 1]; ++t) {
          int s = fwd ? t : brows[t];
          nz += fwd ? (lp[s + 1] - lp[s]) : (up[s + 1] - up[s]);
        }
        return nz;
      };
      // a level goes to the single-CTA run when each of its 32 warps has at
      // most two rows (one dependent load round each); wider levels are one
      // grid launch, whose cost does not grow with the row count
      int rows = ptr[l + 1] - ptr[l];
      int64_t nz = work(l);
      bool narrow = rows <= kRunRows && nz <= kRunEntries;
      if (!narrow) {
        seg.insert(seg.end(), {l, l + 1, lanes_for((double)nz / std::max(1, rows))});
        ++l;
        continue;
      }
      int l1 = l + 1;
      while (l1 < nl) {
        int r = ptr[l1 + 1] - ptr[l1];
        if (r > kRunRows || work(l1) > kRunEntries) break;
        ++l1;
      }
      seg.insert(seg.end(), {l, l1, 1});
      l = l1;
    }
  };
  plan(F.fptr, true, F.fseg);
  plan(F.bptr, false, F.bseg);
}
// levels of the bulk backward sweep start at 0 (rows may point into the tail)
template <class S> void ildl_plan_bwd0(DevFactor<S>& F, const std::vector<int64_t>& up, const std::vector<int>& brows) {
  std::vector<int> seg;
  for (size_t q = 0; q < F.bseg.size(); q += 3) seg.insert(seg.end(), {F.bseg[q], F.bseg[q + 1], F.bseg[q + 2]});
  if (F.bptr.size() > 1 && (F.bseg.empty() || F.bseg[0] != 0)) {
    int64_t nz = 0;
    for (int t = F.bptr[0]; t < F.bptr[1]; ++t) nz += up[brows[t] + 1] - up[brows[t]];
    std::vector<int> s0 = {0, 1, lanes_for((double)nz / std::max(1, F.bptr[1] - F.bptr[0]))};
    s0.insert(s0.end(), seg.begin(), seg.end());
    seg = s0;
  }
  F.bseg = seg;
}

// Coupling blocks of the multilevel form (symAMGsol.c:173-330 applies them
// with CSRMATVEC / CSRMATTVEC): the m rows of a CSR block (row pointers rp[t],
// t < m, global columns) written to y[r0 + t], LANES lanes per row, in the
// outer precision T.  SUB: y[r0 + t] -= sum_q v_q x[c_q]; else
// y[r0 + t] = sum_q v_q x[c_q].  The rows written and the columns read are
// disjoint ranges, so x may alias y.
template <class T, class S, int LANES, bool SUB>
__global__ void __launch_bounds__(WIDE_TPB) couple_kernel(int r0, int m, const int64_t* __restrict__ rp,
                                                         const int* __restrict__ ci, const S* __restrict__ cv,
                                                         const T* x, T* y) {
  pdl_begin();
  const int t = blockIdx.x * (WIDE_TPB / LANES) + (threadIdx.x / LANES);
  const int lane = threadIdx.x % LANES;
  const int r = r0 + t;
  T acc = T(0);
  if (t < m)
    for (int64_t q = rp[t] + lane; q < rp[t + 1]; q += LANES) acc = fma_(cvt<T>(ld_arith(cv + q)), x[ci[q]], acc);
  for (int o = LANES / 2; o > 0; o >>= 1) acc = acc + shfl_xor_any(acc, o);
  if (t < m && lane == 0) y[r] = SUB ? y[r] - acc : acc;
}
template <class T, class S, bool SUB>
static void launch_couple(int lanes, int r0, int m, const int64_t* rp, const int* ci, const S* cv, const T* x, T* y,
                          cudaStream_t s) {
  if (m <= 0) return;
  const int nb = m * lanes / WIDE_TPB + 1;
  if (lanes == 32) launch_k(couple_kernel<T, S, 32, SUB>, dim3(nb), dim3(WIDE_TPB), 0, s, r0, m, rp, ci, cv, x, y);
  else if (lanes == 16) launch_k(couple_kernel<T, S, 16, SUB>, dim3(nb), dim3(WIDE_TPB), 0, s, r0, m, rp, ci, cv, x, y);
  else launch_k(couple_kernel<T, S, 8, SUB>, dim3(nb), dim3(WIDE_TPB), 0, s, r0, m, rp, ci, cv, x, y);
}
// y[r] = yb[r] - t[r] for r in [r0, r0 + m)
template <class T>
__global__ void couple_combine_kernel(int r0, int m, const T* __restrict__ yb, const T* __restrict__ t, T* __restrict__ y) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) y[r0 + i] = yb[r0 + i] - t[r0 + i];
}

template <class T, class S> void ildl_apply(const DevFactor<S>& F, bool spd, const T* b, T* x, cudaStream_t s);

// The multilevel application with coupling blocks: per level l with rows B
// (steps [a, e)) and the later rows C,
//   forward:  y_B = B^{-1} y_B (the level's sub-factor), keep it, y_C -= F^H y_B;
//   backward: t_B = B^{-1} (F y_C), y_B = kept y_B - t_B.
template <class T, class S>
static void ildl_apply_coupled(const DevFactor<S>& F, bool spd, const T* b, T* x, cudaStream_t s) {
  const int n = F.n;
  const int nl = (int)F.lev.size();
  T* y = (T*)F.cy;
  T* yb = (T*)F.cyb;
  T* t = (T*)F.ct;
  launch_k(ildl_gather_kernel<T, T>, dim3(nblk(n)), dim3(TPB), 0, s, n, F.perm, b, y);
  for (int l = 0; l < nl; ++l) {
    const int a = F.lstart[l], e = F.lstart[l + 1];
    ildl_apply<T, S>(F.lev[l], spd, y + a, y + a, s);
    if (l + 1 < nl) {
      CK(cudaMemcpyAsync(yb + a, y + a, sizeof(T) * (size_t)(e - a), cudaMemcpyDeviceToDevice, s));
      launch_couple<T, S, true>(F.fh_lanes[l], e, n - e, F.fhp + F.fh_row0[l], F.fhi, F.fhx, y, y, s);
    }
  }
  for (int l = nl - 2; l >= 0; --l) {
    const int a = F.lstart[l], e = F.lstart[l + 1];
    launch_couple<T, S, false>(F.fp_lanes[l], a, e - a, F.fpp + a, F.fpi, F.fpx, y, t, s);
    ildl_apply<T, S>(F.lev[l], spd, t + a, t + a, s);
    launch_k(couple_combine_kernel<T>, dim3(nblk(e - a)), dim3(TPB), 0, s, a, e - a, (const T*)yb, (const T*)t, y);
  }
  launch_k(ildl_scatter_kernel<T, T>, dim3(nblk(n)), dim3(TPB), 0, s, n, F.perm, (const T*)y, x);
}

template <class T, class S> void ildl_apply(const DevFactor<S>& F, bool spd, const T* b, T* x, cudaStream_t s) {
  using A = typename Arith<S>::type;
  const int n = F.n;
  if (F.coupled) {
    ildl_apply_coupled<T, S>(F, spd, b, x, s);
    return;
  }
  launch_k(ildl_gather_kernel<T, A>, dim3(nblk(n)), dim3(TPB), 0, s, n, F.orig, b, F.y);
  auto sweep = [&](const std::vector<int>& seg, const std::vector<int>& ptr, const int* dptr, const int* rows,
                   const int64_t* rp, const int* ci, const S* cv) {
    for (size_t q = 0; q < seg.size(); q += 3) {
      int l0 = seg[q], l1 = seg[q + 1];
      if (seg[q + 2] == 1) {
        launch_k(ildl_run_kernel<S, A>, dim3(1), dim3(RUN_TPB), 0, s, l0, l1, dptr, rows, rp, ci, cv, F.y);
      } else {
        launch_wide<S, A>(seg[q + 2], ptr[l0], ptr[l0 + 1], rows, rp, ci, cv, F.y, s);
      }
    }
  };
  sweep(F.fseg, F.fptr, F.dfptr, nullptr, F.lp, F.li, F.lx);
  const bool dense = !F.blocks.empty(), levels = F.m_tail > 0 && !dense;
  auto ext = [&](int m, int s0, const int64_t* rp, const int* ci, const S* cv, int64_t entries, A* out) {
    launch_ext<S, A>(lanes_for((double)entries / std::max(1, m)), m, s0, rp, ci, cv, F.y, out, entries, s);
  };
  const size_t tsm = levels ? std::max(tail_smem_bytes<A>(F.m_tail, (int)F.tfptr.size() - 1, false),
                                       tail_smem_bytes<A>(F.m_tail, (int)F.tbptr.size() - 1, true))
                            : 0;
  if (levels) ensure_tail_smem<S, A>(tsm);
  if (dense) {
    for (const auto& B : F.blocks) {
      A* yb = F.y + B.s0;
      if (B.nt > 0) {
        // right-hand side into xb, then y_B = T xb
        ext(B.m, B.s0, B.ep, B.ei, B.ev, B.nfe, F.xb);
        launch_tri<S, A>(B.nitf, B.tcl, true, (const int4*)B.itf, B.tf, (const A*)F.xb, B.m, yb, s);
      } else if (B.nfe > 0) {
        ext(B.m, B.s0, B.ep, B.ei, B.ev, B.nfe, yb);
      }
    }
  } else if (levels) {
    ext(F.m_tail, F.s_tail, F.tep, F.tei, F.tev, 8 * (int64_t)F.m_tail, F.y + F.s_tail);
    launch_k(tail_run_kernel<S, A>, dim3(1), dim3(RUN_TPB), tsm, s, F.m_tail, F.s_tail, (int)F.tfptr.size() - 1, F.dtfptr, nullptr,
                                                 F.tip, F.tii, F.tiv, F.y);
  }
  launch_k(ildl_dsolve_kernel<S, A>, dim3(nblk(n)), dim3(TPB), 0, s, n, F.blk, F.partner, spd ? F.av : F.dv, spd ? F.aof : F.dof, F.y);
  if (dense) {
    for (auto it = F.blocks.rbegin(); it != F.blocks.rend(); ++it) {
      const auto& B = *it;
      A* yb = F.y + B.s0;
      if (B.nt > 0) {
        ext(B.m, B.s0, B.bp, B.bi, B.bv, B.nbe, F.xb);
        launch_tri<S, A>(B.nitb, B.tcl, false, (const int4*)B.itb, B.tb, (const A*)F.xb, B.m, yb, s);
      } else if (B.nbe > 0) {
        ext(B.m, B.s0, B.bp, B.bi, B.bv, B.nbe, yb);
      }
    }
  } else if (levels) {
    launch_k(tail_run_kernel<S, A>, dim3(1), dim3(RUN_TPB), tsm, s, F.m_tail, F.s_tail, (int)F.tbptr.size() - 1, F.dtbptr, F.tbrows,
                                                 F.tbp, F.tbi, F.tbv, F.y);
  }
  sweep(F.bseg, F.bptr, F.dbptr, F.brows, F.up, F.ui, F.ux);
  launch_k(ildl_scatter_kernel<T, A>, dim3(nblk(n)), dim3(TPB), 0, s, n, F.orig, F.y, x);
}

// The captured application reads b and writes x where the caller has them: its
// first kernel (the gather) and its last (the scatter) are pointed at new
// vectors when those differ from the last call's, about twice per solve.
// Copying them to and from fixed vectors cost two 4 us copies per application.
// us per application with them -> without (GB300): Anderson 16^3 24.6 -> 14.4,
// 28^3 66.4 -> 57.8, Laplacian 20^3 65.8 -> 58.2.
template <class T, class S> void ildl_apply_graph(DevFactor<S>& F, bool spd, const T* b, T* x, cudaStream_t s) {
  using A = typename Arith<S>::type;
  const int g = spd ? 1 : 0;
  if (!F.graph[g]) {
    auto smem = [](const DevFactor<S>& D) {
      if (D.m_tail > 0 && D.blocks.empty())
        ensure_tail_smem<S, A>(std::max(tail_smem_bytes<A>(D.m_tail, (int)D.tfptr.size() - 1, false),
                                        tail_smem_bytes<A>(D.m_tail, (int)D.tbptr.size() - 1, true)));
    };
    smem(F);
    for (const auto& D : F.lev) smem(D);
    cudaGraph_t gr;
    CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    ildl_apply<T, S>(F, spd, b, x, s);
    CK(cudaStreamEndCapture(s, &gr));
    F.graph_def[g] = gr;  // the nodes below are its nodes
    size_t nn = 0, nr = 1, ne = 0;
    CK(cudaGraphGetNodes(gr, nullptr, &nn));
    F.graph_kernels[g] = (long long)nn;
    CK(cudaGraphGetRootNodes(gr, &F.graph_in[g], &nr));
    // the last kernel: the node no edge leaves
    CK(cudaGraphGetEdges(gr, nullptr, nullptr, nullptr, &ne));
    std::vector<cudaGraphNode_t> from(ne), to(ne), all(nn);
    std::vector<cudaGraphEdgeData> data(ne);
    CK(cudaGraphGetEdges(gr, from.data(), to.data(), data.data(), &ne));
    CK(cudaGraphGetNodes(gr, all.data(), &nn));
    int last = 0;
    for (cudaGraphNode_t v : all)
      if (std::find(from.begin(), from.end(), v) == from.end()) {
        F.graph_out[g] = v;
        ++last;
      }
    if (nr != 1 || last != 1) throw std::runtime_error("the captured application is not a chain of kernels");
    CK(cudaGraphInstantiate(&F.graph[g], gr, 0));
    F.graph_b[g] = b;
    F.graph_x[g] = x;
  }
  auto point = [&](cudaGraphNode_t node, void** args) {
    cudaKernelNodeParams p = {};
    CK(cudaGraphKernelNodeGetParams(node, &p));
    p.kernelParams = args;
    p.extra = nullptr;
    CK(cudaGraphExecKernelNodeSetParams(F.graph[g], node, &p));
  };
  const int* order = F.coupled ? F.perm : F.orig;
  void* work = F.coupled ? F.cy : (void*)F.y;
  int n = F.n;
  if (F.graph_b[g] != (const void*)b) {
    void* args[] = {&n, &order, &b, &work};
    point(F.graph_in[g], args);
    F.graph_b[g] = b;
  }
  if (F.graph_x[g] != (void*)x) {
    void* args[] = {&n, &order, &work, &x};
    point(F.graph_out[g], args);
    F.graph_x[g] = x;
  }
  CK(cudaGraphLaunch(F.graph[g], s));
  g_launches += F.graph_kernels[g];
}

// ------------------------------------------------------- instantiations ----
#define JD_INST_T(T)                                                                               \
  template bool sell_from_triangle<T>(int, const int*, const int*, const void*, void*, int64_t*, unsigned long long*, \
                                      const std::function<void(int64_t, int**, T**)>&, cudaStream_t); \
  template void spmv<T>(const SellMatrix<T>&, const T*, T*, cudaStream_t);                         \
  template void axpy<T>(long, T, const T*, T*, cudaStream_t);                                      \
  template void gemv_dot<T>(long, int, const T*, long, const T*, T*, const T*, T*, T*, cudaStream_t, const T*, int, \
                            T*, const T*, const T*, double*);                                     \
  template bool inner_one_ok<T>(long, int, bool);                                                 \
  template int inner_one<T>(const SellMatrix<T>&, const SellMatrix<T>*, int, const T*, const T*, T*, T*, T*, double, bool, \
                            bool, T*, const T*, T*, T*, double*, unsigned*, OneState&, cudaStream_t); \
  template void cg_direction<T>(long, const T*, const double*, bool, T*, T*, cudaStream_t);           \
  template void spmv_shift<T>(const SellMatrix<T>&, const SellMatrix<T>*, double, const T*, T*, T*, cudaStream_t); \
  template void cg_residual<T>(long, const double*, const T*, T*, T*, const T*, int, T*, T*, cudaStream_t); \
  template void cg_iterate<T>(long, bool, bool, double, double, const T*, T*, T*, double, const T*, T*, cudaStream_t); \
  template void axpy_dev<T>(long, const T*, double, const T*, T*, cudaStream_t);                  \
  template void scal<T>(long, double, T*, cudaStream_t);                                           \
  template void fill<T>(long, T, T*, cudaStream_t);                                                \
  template void mdot<T>(long, int, const T*, long, const T*, T*, T*, cudaStream_t, const T*);      \
  template void gemv_dev<T>(long, int, double, const T*, long, const T*, double, T*, cudaStream_t, T*);      \
  template void ritz<T>(long, int, const T*, const T*, const T*, long, const T*, double, T*, T*, T*, T*, T*, cudaStream_t); \
  template void gemv_val<T>(long, int, double, const T*, long, const T*, double, T*, cudaStream_t);          \
  template void rmult<T>(long, int, int, const T*, long, const T*, T*, cudaStream_t);              \
  template void diagsolve<T>(long, const double*, const T*, T*, cudaStream_t);
JD_INST_T(double)
JD_INST_T(zc)
#define JD_INST_F(T, S)                                                                          \
  template void ildl_apply<T, S>(const DevFactor<S>&, bool, const T*, T*, cudaStream_t);          \
  template void ildl_apply_graph<T, S>(DevFactor<S>&, bool, const T*, T*, cudaStream_t);          \
  template void ildl_plan<S>(DevFactor<S>&, const std::vector<int64_t>&, const std::vector<int64_t>&, \
                             const std::vector<int>&);                                          \
  template void ildl_plan_bwd0<S>(DevFactor<S>&, const std::vector<int64_t>&, const std::vector<int>&); \
  template bool tri_cluster16_ok<S, typename Arith<S>::type>();
JD_INST_F(double, double)
JD_INST_F(double, float)
JD_INST_F(double, __nv_bfloat16)
JD_INST_F(zc, zc)
JD_INST_F(zc, cc)
JD_INST_F(zc, bc)

}  // namespace k
}  // namespace jdg
