// One bond split on one CTA, and the split's reciprocal square roots, as
// functions of host arrays: what the GPU tests of csrc/split.cuh call.
#include <vector>

#include "../../oqupy_gb300/csrc/engine.h"
#include "../../oqupy_gb300/csrc/split.cuh"

namespace otb {

constexpr int PROBE_SMEM = 88 * 1024;

// A (R x N, column-major) -> the kept columns of W, in order, with their norms
// and meta = (kept, flip, status, sweeps).
template <typename T>
__global__ void __launch_bounds__(256)
    split_probe_kernel(const zc* A, int R, int N, double epsrel, float qr_cut, unsigned char* work, long long wcap,
                       zc* W, double* norm, int* meta) {
  typedef QA<T> Q;
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ SplitShared sh;
  typename Q::E* src = reinterpret_cast<typename Q::E*>(work + wcap * 16);
  for (int i = threadIdx.x; i < R * N; i += blockDim.x) src[i] = Q::from(A[i]);
  __syncthreads();
  SplitBufs b;
  b.Wg = work;
  b.Xg = work + wcap * 48;
  b.Mg = work + wcap * 64;
  b.bkg = work + wcap * 96;
  b.smem = dsm;
  b.smem_bytes = PROBE_SMEM;
  const PlainSource<T> s{src, R, false};
  const SplitOut<T> o = oriented_split<T>(s, R, N, epsrel, qr_cut, b, sh);
  const int ld = o.flip ? N : R;
  const double scale = ldexp(1.0, o.e);
  for (int i = threadIdx.x; i < ld * o.kk; i += blockDim.x) {
    const int j = i / ld, r = i - j * ld;
    W[i] = cscale(Q::to(o.W[(size_t)sh.book.perm[j] * ld + r]), scale);
  }
  for (int j = threadIdx.x; j < o.kk; j += blockDim.x) norm[j] = sh.book.norm[sh.book.perm[j]];
  if (threadIdx.x == 0) {
    meta[0] = o.kk;
    meta[1] = o.flip;
    meta[2] = sh.jsh.status;
    meta[3] = sh.jsh.sweeps;
  }
}

__global__ void rsqrt_probe_kernel(const double* x, double* d, double* f, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  d[i] = QA<double>::rsqrt(x[i]);
  f[i] = ff_to(QA<ff>::rsqrt(ff_from(x[i])));
}

struct Dev {
  void* p = nullptr;
  explicit Dev(size_t bytes) { cudaMalloc(&p, bytes); }
  ~Dev() { cudaFree(p); }
};

template <typename T>
static int run_split(const double* A, int R, int N, double epsrel, double qr_cut, double* W, double* norm, int* meta) {
  const long long wcap = (long long)R * R;
  Dev a((size_t)R * N * 16), work((size_t)wcap * 96 + QR_BOOK_BYTES), w((size_t)R * N * 16), s(N * 8), m(16);
  if (!a.p || !work.p || !w.p || !s.p || !m.p) return -1;
  cudaMemcpy(a.p, A, (size_t)R * N * 16, cudaMemcpyHostToDevice);
  cudaMemset(m.p, 0, 16);
  cudaFuncSetAttribute(split_probe_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, PROBE_SMEM);
  split_probe_kernel<T><<<1, 256, PROBE_SMEM>>>((const zc*)a.p, R, N, epsrel, (float)qr_cut, (unsigned char*)work.p,
                                                wcap, (zc*)w.p, (double*)s.p, (int*)m.p);
  cudaMemcpy(W, w.p, (size_t)R * N * 16, cudaMemcpyDeviceToHost);
  cudaMemcpy(norm, s.p, (size_t)N * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(meta, m.p, 16, cudaMemcpyDeviceToHost);
  return (int)cudaGetLastError();
}

}  // namespace otb

using namespace otb;

extern "C" int split_probe(int mixed, const double* A, int R, int N, double epsrel, double qr_cut, double* W,
                           double* norm, int* meta) {
  if (N < 1 || R < N || R > SPLIT_NMAX) return -1;
  return mixed ? run_split<ff>(A, R, N, epsrel, qr_cut, W, norm, meta)
               : run_split<double>(A, R, N, epsrel, qr_cut, W, norm, meta);
}

extern "C" int rsqrt_probe(const double* x, double* d, double* f, int n) {
  Dev a((size_t)n * 8), b((size_t)n * 8), c((size_t)n * 8);
  if (!a.p || !b.p || !c.p) return -1;
  cudaMemcpy(a.p, x, (size_t)n * 8, cudaMemcpyHostToDevice);
  rsqrt_probe_kernel<<<(n + 255) / 256, 256>>>((const double*)a.p, (double*)b.p, (double*)c.p, n);
  cudaMemcpy(d, b.p, (size_t)n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(f, c.p, (size_t)n * 8, cudaMemcpyDeviceToHost);
  return (int)cudaGetLastError();
}
