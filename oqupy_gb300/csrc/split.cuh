// Truncated bond split of one CTA, shared by the TEMPO step and the PT-TEMPO
// build.
//
// oriented_split() reads the oriented matrix A (R x N, R >= N) through an
// accessor -- key(r, c): magnitude key, exponent(key): its power of two,
// load(X, R, N, e): X = A 2^-e in the split's arithmetic -- and runs the
// QR-preconditioned Jacobi (qr.cuh; plain Jacobi, jacobi.cuh, below 8
// columns).
#pragma once

#include "qr.cuh"

namespace otb {

typedef cx<double> zc;

constexpr int QR_MIN_COLS = 8;

// The splits' arithmetic of a precision form.
template <bool MIXED>
struct StepType {
  typedef double T;
};
template <>
struct StepType<true> {
  typedef ff T;
};

struct SplitShared {
  SplitBook book;
  JacobiShared jsh;
  unsigned mag[32];   // largest magnitudes by warp
};

// Per-CTA working storage: global matrices of wcap 16-byte elements and the
// dynamic shared memory.
struct SplitBufs {
  void* Wg;             // spare matrix (the QR's row factor when it does not fit in shared memory)
  void* Xg;             // working matrix when it does not fit in shared memory
  void* Mg;             // FP64: two more, for the orthogonalisation's products
  unsigned char* bkg;   // QR bookkeeping of more than 383 columns when shared memory is too small
  unsigned char* smem;
  int smem_bytes;
};

// Result of oriented_split: W's columns book.perm[0 .. kk) are, with sigma =
// book.norm[...] and all of W over `scale`,
//   flip false: A V Sigma (R x N, ld R);   flip true: A^H U Sigma (N x k, ld N)
// for the oriented A (R x N).
template <typename T>
struct SplitOut {
  typename QA<T>::E* W;
  int kk;
  int e;       // scale = 2^e
  bool flip;
};

template <typename T, class Acc>
__device__ __forceinline__ SplitOut<T> oriented_split(const Acc& A, int R, int N, double epsrel, float qr_delta,
                                                      const SplitBufs& b, SplitShared& sh) {
  typedef QA<T> Q;
  typedef typename Q::E E;
  const int tid = threadIdx.x, nt = blockDim.x;
  SplitOut<T> o;
  const size_t xbytes = (size_t)R * N * sizeof(E);
  const bool x_shared = xbytes <= (size_t)b.smem_bytes;
  E* X = x_shared ? reinterpret_cast<E*>(b.smem) : reinterpret_cast<E*>(b.Xg);
  // power-of-two scale from the largest magnitude (exact)
  unsigned mx = 0u;
  for (int idx = tid; idx < R * N; idx += nt) {
    const int c = idx / R, r = idx - c * R;
    mx = max(mx, A.key(r, c));
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((tid & 31) == 0) sh.mag[tid >> 5] = mx;
  __syncthreads();
  mx = (tid & 31) < (nt >> 5) ? sh.mag[tid & 31] : 0u;
  mx = __reduce_max_sync(0xffffffffu, mx);
  o.e = A.exponent(mx);
  A.load(X, R, N, o.e);
  __syncthreads();
  const double scale = ldexp(1.0, o.e);
  o.flip = N >= QR_MIN_COLS;
  if (o.flip) {
    const size_t used = x_shared ? xbytes : 0;
    o.kk = qr_jacobi_truncate<T>(X, x_shared, R, N, scale, reinterpret_cast<E*>(b.Wg), reinterpret_cast<E*>(b.Mg),
                                 b.smem + used, (size_t)b.smem_bytes - used, b.bkg, epsrel, qr_delta, &sh.book,
                                 &sh.jsh, &o.W);
    return o;
  }
  const int sw64 = jacobi_norms<T>(X, R, N, R, scale, sh.book.norm, &sh.jsh);
  o.kk = jacobi_rank(N, epsrel, sh.book.norm, sh.book.perm, &sh.jsh, sw64, 0.0, scale);
  o.W = X;
  return o;
}

// Accessor of the oriented matrix over a plain array of the split's own
// element type: A(r, c) = src[c * lds + r], or its conjugate transpose
// A(r, c) = conj(src[r * lds + c]).
template <typename T>
struct PlainSource {
  typedef QA<T> Q;
  typedef typename Q::E E;
  const E* src;
  int lds;
  bool trans;
  __device__ __forceinline__ E at(int r, int c) const {
    return trans ? src[(size_t)r * lds + c] : src[(size_t)c * lds + r];
  }
  __device__ __forceinline__ unsigned key(int r, int c) const { return Q::mag_key(at(r, c)); }
  __device__ __forceinline__ int exponent(unsigned key) const { return Q::key_exponent(key); }
  __device__ __forceinline__ void load(E* X, int R, int N, int e) const {
    const typename Q::P p2 = Q::pow2(-e);
    for (int idx = threadIdx.x; idx < R * N; idx += blockDim.x) {
      const int c = idx / R, r = idx - c * R;
      const E x = Q::ldexpE(at(r, c), p2);
      X[idx] = trans ? Q::conj(x) : x;
    }
  }
};

}  // namespace otb
