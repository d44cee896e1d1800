// Rank-revealing QR + one-sided Jacobi on the reduced factor: the truncated
// bond split of both precision forms for splits of >= 8 columns (smaller
// splits run plain Jacobi, jacobi.cuh).
//
// Replaces, like jacobi.cuh, the truncated SVD that the reference obtains
// from tensornetwork's split_node_full_svd(max_truncation_err=epsrel,
// relative=True) (oqupy/backends/node_array.py:262-268, 285-291, 541-547),
// with the rank rule chi = #{i : sqrt(sum_{j>=i} s_j^2) > epsrel * s_0}
// (oqupy/mps_mpo.py:452-457).
//
// The oriented matrix A (R x N, R >= N) is factorised A P = Q R with column
// pivoting, stopped at the first step k whose remaining block has Frobenius
// norm below delta times the largest initial column norm.  One-sided Jacobi
// then orthogonalises the columns of Z = P R[0:k, :]^H (N x k): the pivoted R
// is graded, so Z converges in few sweeps, and it has only k columns.  With
// Z V = W orthogonal, A ~= (Q V) Sigma (W / Sigma)^H, so W = A^H U Sigma: the
// caller receives the conjugate-side factor (N x k, ld N).  The dropped
// block's squared norm belongs to the tail of every kept index and is added
// to the tail sums, so the rank decision is that of the full decomposition up
// to delta.
//
// Q itself is never used, so R comes from modified Gram-Schmidt: R is as
// accurate as the Householder one (backward stable), the projection of a
// column on the pivot column needs no reflector scalars -- the coefficient
// conj(p) . x / |p|^2 takes one reciprocal square root, evaluated while the
// inner products are being formed -- and row i of R is just those inner
// products.
#pragma once

#include <climits>

#include "orthogonal.cuh"

namespace otb {

constexpr int SPLIT_NMAX = 1152;  // max columns of a split (D * chi_cap <= 1152)

// The split's per-column results and, while the QR runs, its bookkeeping.
struct SplitBook {
  double norm[SPLIT_NMAX];
  int perm[SPLIT_NMAX];
};

// QR bookkeeping (36 bytes a column): squared norms of the unchosen columns
// and their FP32 keys by list position, the list itself (column of every
// position), all double-buffered by step parity, and the inverse pivot norms.
struct QrBook {
  unsigned char* p;
  int N;
  template <typename S>
  __device__ S* n2(int par) const { return reinterpret_cast<S*>(p) + par * N; }
  template <typename S>
  __device__ S* rinv() const { return reinterpret_cast<S*>(p) + 2 * N; }
  __device__ float* key(int par) const { return reinterpret_cast<float*>(p + (size_t)24 * N) + par * N; }
  __device__ short* list(int par) const { return reinterpret_cast<short*>(p + (size_t)32 * N) + par * N; }
};
__host__ __device__ constexpr size_t qr_book_bytes(int N) { return (size_t)36 * N + 16; }

// Default relative cut of the QR (the remaining block's Frobenius norm over
// the largest initial column norm) for each arithmetic.
__device__ __forceinline__ float qr_default_delta(bool ffarith, double epsrel) {
  return ffarith ? (float)fmin(1e-3 * epsrel, 1e-9) : 1e-14f;
}

// Lanes per column of a QR step, from the operand's shape only (an instance's
// rounding must not depend on the launch shape or on the batch it is in).  As
// for the Jacobi pairs, wider groups repeat a column's scalar work in more
// warps: few lanes while many columns are left, more once they run out.
__device__ __forceinline__ int qr_group(int rows, int cols) {
  int G = rows > 160 ? 32 : (rows > 64 ? 16 : 8);
  while (G < 32 && G * cols <= 96 && rows > 2 * G) G <<= 1;
  return G;
}

// About 1 / (|v| |c|) from squared norms; columns below 1e-15 (zero columns
// among them) count as 1e-15, which only makes the bound a loose one.
__device__ __forceinline__ float inverse_bound(float v2, float c2) {
  return rsqrt_est(fmaxf(v2, 1e-30f)) * rsqrt_est(fmaxf(c2, 1e-30f));
}

// One Gram-Schmidt projection by a group of G lanes (lane gl): (wr, wi) =
// v^H c, c <- c - v beta (wr + i wi), s2 = |c|^2 (of the new column; all
// results in every lane).  rb is about 1 / (|v| |c|).  RC rows a lane at a time in registers (all of its
// rows with ALL: R <= RC G), so that the rows' chains overlap.
template <typename T, int G, int RC, bool ALL>
__device__ __forceinline__ void project_rc(const typename QA<T>::E* v, typename QA<T>::E* c, int R, int gl,
                                           bool act, typename QA<T>::S beta, float rb, typename QA<T>::S& wr,
                                           typename QA<T>::S& wi, typename QA<T>::S& s2) {
  typedef QA<T> Q;
  typedef typename Q::E E;
  wr = wi = s2 = Q::zero();
  E a[RC], x[RC];
  for (int r0 = gl; r0 < (ALL ? gl + 1 : R); r0 += RC * G) {
#pragma unroll
    for (int q = 0; q < RC; ++q) {
      const bool in = act && r0 + q * G < R;
      a[q] = in ? v[r0 + q * G] : Q::zeroE();
      x[q] = in ? c[r0 + q * G] : Q::zeroE();
    }
#pragma unroll
    for (int q = 0; q < RC; ++q) Q::dotj(wr, wi, a[q], x[q]);
  }
  Q::template dot_sum<G>(wr, wi, rb);
  const typename Q::S bx = Q::mul(beta, wr), by = Q::mul(beta, wi);
  for (int r0 = gl; r0 < (ALL ? gl + 1 : R); r0 += RC * G) {
#pragma unroll
    for (int q = 0; q < RC; ++q) {
      if (!ALL) {
        const bool in = act && r0 + q * G < R;
        a[q] = in ? v[r0 + q * G] : Q::zeroE();
        x[q] = in ? c[r0 + q * G] : Q::zeroE();
      }
    }
#pragma unroll
    for (int q = 0; q < RC; ++q) {
      x[q] = Q::sub_scaled(x[q], a[q], bx, by);
      s2 = Q::abs2_acc(x[q], s2);
    }
#pragma unroll
    for (int q = 0; q < RC; ++q)
      if (act && r0 + q * G < R) c[r0 + q * G] = x[q];
  }
  s2 = Q::fin(Q::template group_sum<G>(s2));
}

template <typename T>
__device__ __forceinline__ void project(const typename QA<T>::E* v, typename QA<T>::E* c, int R, int G, int gl,
                                        bool act, typename QA<T>::S beta, float rb, typename QA<T>::S& wr,
                                        typename QA<T>::S& wi, typename QA<T>::S& s2) {
  if (G == 8) {
    if (R <= 32)
      project_rc<T, 8, 4, true>(v, c, R, gl, act, beta, rb, wr, wi, s2);
    else
      project_rc<T, 8, 4, false>(v, c, R, gl, act, beta, rb, wr, wi, s2);
  } else if (G == 16) {
    if (R <= 32)
      project_rc<T, 16, 2, true>(v, c, R, gl, act, beta, rb, wr, wi, s2);
    else if (R <= 64)
      project_rc<T, 16, 4, true>(v, c, R, gl, act, beta, rb, wr, wi, s2);
    else
      project_rc<T, 16, 4, false>(v, c, R, gl, act, beta, rb, wr, wi, s2);
  } else {
    if (R <= 64)
      project_rc<T, 32, 2, true>(v, c, R, gl, act, beta, rb, wr, wi, s2);
    else
      project_rc<T, 32, 4, false>(v, c, R, gl, act, beta, rb, wr, wi, s2);
  }
}

// The FP64 form of a step on the columns of X (R rows): with v the pivot column,
// c <- c - v (v^H c) / |v|^2 for the `nrest` columns list[t] (list[t + 1] from
// t = pos on), by a group of G lanes each.  out[j ostride] receives column j's
// inner product v^H c, nkey[t] / nlist[t] its new FP32 squared norm and index.
// In between, the last warp forms |v|^2 in full: *diag and *rinv receive
// |v|^2 and 1 / |v|, all others 1 / |v|^2 through *beta_sh.  Ends with a
// barrier.
//
// The columns' own squared norms only rank them and decide the stop, so FP32
// is enough for all but the pivot's: against project(), which keeps them in the
// columns' arithmetic and has every warp form the pivot's reciprocal, a column
// takes 8 instead of 10 multiply-adds an element, a group two reductions less,
// for one barrier more.  48 instances of splits ~77 x 31: 25100 instead of
// 35300 clocks a step, bound by the FP64 pipe in both.  Double-float columns
// keep project(): with one instruction a clock the barrier and the reloads cost
// what the norms save (splits of ~77 x 35: 16600 and 15600 clocks a step).
struct GsStep {
  cx<double>* X;
  const cx<double>* v;
  cx<double>*out, *diag;
  double *rinv, *beta_sh;
  const float* key;
  const short* list;
  float* nkey;
  short* nlist;
  size_t ostride;
  int R, nrest, pos;
  float v2;
};

// RC rows a lane at a time.  Both halves read the columns (an element's loads
// are hidden behind its multiply-adds, 64 clocks each); the inner products wait
// in `out`.
template <int G, int RC>
__device__ __forceinline__ void gs_columns(const GsStep& g) {
  typedef QA<double> Q;
  typedef cx<double> E;
  const int gl = threadIdx.x & (G - 1), group = threadIdx.x / G, ngroups = blockDim.x / G;
  const int first = (int)(threadIdx.x & ~31u) / G;   // the warp's first group
  for (int tb = 0; tb + first < g.nrest; tb += ngroups) {
    const int t = tb + group;
    const bool act = t < g.nrest;
    const int p = act ? t + (t >= g.pos ? 1 : 0) : 0;
    const int j = g.list[p];
    const E* c = g.X + (size_t)j * g.R;
    double wr = 0.0, wi = 0.0;
    for (int r0 = gl; r0 < g.R; r0 += RC * G) {
      E a[RC], x[RC];
#pragma unroll
      for (int q = 0; q < RC; ++q) {
        const bool in = act && r0 + q * G < g.R;
        a[q] = in ? g.v[r0 + q * G] : Q::zeroE();
        x[q] = in ? c[r0 + q * G] : Q::zeroE();
      }
#pragma unroll
      for (int q = 0; q < RC; ++q) Q::dotj(wr, wi, a[q], x[q]);
    }
    __syncwarp();
    Q::dot_sum<G>(wr, wi, inverse_bound(g.v2, g.key[p]));
    if (act && gl == 0) g.out[j * g.ostride] = mk<double>(wr, wi);
  }
  __syncthreads();
  const double beta = *g.beta_sh;
  for (int tb = 0; tb + first < g.nrest; tb += ngroups) {
    const int t = tb + group;
    const bool act = t < g.nrest;
    const int j = g.list[act ? t + (t >= g.pos ? 1 : 0) : 0];
    E* c = g.X + (size_t)j * g.R;
    float s2 = 0.f;
    if (act) {
      const E w = g.out[j * g.ostride];
      const double bx = Q::mul(beta, w.x), by = Q::mul(beta, w.y);
      for (int r0 = gl; r0 < g.R; r0 += RC * G) {
        E x[RC];
#pragma unroll
        for (int q = 0; q < RC; ++q) {
          const bool in = r0 + q * G < g.R;
          x[q] = in ? Q::sub_scaled(c[r0 + q * G], g.v[r0 + q * G], bx, by) : Q::zeroE();
          s2 = Q::abs2_32(x[q], s2);
        }
#pragma unroll
        for (int q = 0; q < RC; ++q)
          if (r0 + q * G < g.R) c[r0 + q * G] = x[q];
      }
    }
    __syncwarp();
#pragma unroll
    for (int off = G >> 1; off > 0; off >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, off, 32);
    if (act && gl == 0) {
      g.nkey[t] = s2;
      g.nlist[t] = (short)j;
    }
  }
}

__device__ __forceinline__ void gs_step(const GsStep& g) {
  typedef QA<double> Q;
  if (threadIdx.x >> 5 == (blockDim.x >> 5) - 1) {
    double acc = 0.0;
    for (int r = threadIdx.x & 31; r < g.R; r += 32) acc = Q::abs2_acc(g.v[r], acc);
    __syncwarp();
    acc = Q::group_sum<32>(acc);
    const double ri = Q::rsqrt(acc);
    if ((threadIdx.x & 31) == 0) {
      *g.beta_sh = Q::mul(ri, ri);
      *g.rinv = ri;
      *g.diag = Q::realE(acc);
    }
  }
  const int G = qr_group(g.R, g.nrest);
  if (G == 8)
    gs_columns<8, 3>(g);
  else if (G == 16)
    gs_columns<16, 3>(g);
  else
    gs_columns<32, 3>(g);
  __syncthreads();
}

// Pivoted Gram-Schmidt QR of X (R x N, column-major ld R; destroyed).
// Returns k and writes Z (N x k, ld N): Z[q, i] = conj(R[i, q]), zero where
// column q was chosen before step i; Z's storage holds N x N.  *tail2 is the
// remaining squared mass at the stop (0 when all N steps ran).
//
// One __syncthreads per step, no column moves: every warp finds the pivot
// (largest squared norm, first list position on ties) and the remaining mass
// from the list's keys; every column's group forms its inner product with the
// pivot column, updates the column and leaves its new squared norm, key and
// list entry in the other buffer.  A step is bound by the chain key ->
// pivot -> inner product -> reduction -> update (and, per CTA, by the
// double-float or FP64 issue rate while many columns are left).  Against the
// Householder form it replaces (reflector norm and scalars by every warp,
// three dependent reductions per step) a step of a 45 x 22 double-float
// operand takes 5700 instead of 8000 clocks, of a 57 x 26 FP64 one 14000
// instead of 22000.
template <typename T>
__device__ int pivoted_qr(typename QA<T>::E* X, int R, int N, float delta, const QrBook& bk, typename QA<T>::E* Z,
                          float* tail2) {
  typedef QA<T> Q;
  typedef typename Q::E E;
  typedef typename Q::S S;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane32 = tid & 31, warp = tid >> 5, nw = nt >> 5;
  for (int j = warp; j < N; j += nw) {
    S acc = Q::zero();
    const E* c = X + (size_t)j * R;
    for (int r = lane32; r < R; r += 32) acc = Q::abs2_acc(c[r], acc);
    acc = Q::fin(Q::template group_sum<32>(acc));
    if (lane32 == 0) {
      bk.n2<S>(0)[j] = acc;
      bk.key(0)[j] = Q::tof(acc);
      bk.list(0)[j] = (short)j;
    }
  }
  for (int idx = tid; idx < N * N; idx += nt) Z[idx] = Q::zeroE();
  __syncthreads();
  float cut = 0.f, t2 = 0.f;
  int k = N;
  for (int i = 0; i < N; ++i) {
    const int n = N - i, cur = i & 1, nxt = cur ^ 1;
    const float* key = bk.key(cur);
    const short* list = bk.list(cur);
    float bv = 0.f, sum = 0.f;
    int bq = INT_MAX;
    for (int q = lane32; q < n; q += 32) {
      const float v = key[q];
      sum += v;
      if (bq == INT_MAX || v > bv) {
        bv = v;
        bq = q;
      }
    }
    const unsigned best = __reduce_max_sync(0xffffffffu, __float_as_uint(bv));
    const int pos = (int)__reduce_min_sync(0xffffffffu, __float_as_uint(bv) == best ? (unsigned)bq : (unsigned)INT_MAX);
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (i == 0) {
      cut = delta * delta * __uint_as_float(best);
    } else if (sum < cut) {
      k = i;
      t2 = sum;
      break;
    }
    const int p = list[pos];
    if constexpr (!Q::kFF) {
      GsStep g;
      g.X = X;
      g.v = X + (size_t)p * R;
      g.out = Z + (size_t)i * N;
      g.ostride = 1;
      g.diag = g.out + p;
      g.rinv = bk.rinv<S>() + i;
      g.beta_sh = bk.n2<S>(0);
      g.key = key;
      g.list = list;
      g.nkey = bk.key(nxt);
      g.nlist = bk.list(nxt);
      g.R = R;
      g.nrest = n - 1;
      g.pos = pos;
      g.v2 = __uint_as_float(best);
      gs_step(g);
    } else {
      const S np = bk.n2<S>(cur)[pos];
      const S ri = Q::rsqrt(np);
      const S beta = Q::mul(ri, ri);
      if (tid == 0) {
        bk.rinv<S>()[i] = ri;
        Z[(size_t)i * N + p] = Q::realE(np);
      }
      const E* v = X + (size_t)p * R;
      const int nrest = n - 1;
      const int G = qr_group(R, nrest);
      const int gl = tid & (G - 1), group = tid / G, ngroups = nt / G;
      for (int tb = 0; tb < nrest; tb += ngroups) {
        if (tb + (warp * 32) / G >= nrest) break;   // no column left for this warp
        const int t = tb + group;
        const bool act = t < nrest;
        const int q = act ? t + (t >= pos ? 1 : 0) : pos;
        const int j = list[q];
        const float rb = inverse_bound(__uint_as_float(best), key[q]);
        E* cj = X + (size_t)j * R;
        S wr, wi, s2;
        project<T>(v, cj, R, G, gl, act, beta, rb, wr, wi, s2);
        if (act && gl == 0) {
          bk.n2<S>(nxt)[t] = s2;
          bk.key(nxt)[t] = Q::tof(s2);
          bk.list(nxt)[t] = (short)j;
          E z;
          z.x = wr;
          z.y = wi;
          Z[(size_t)i * N + j] = z;
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();   // a stop at step k leaves warps that may still be reading the keys
  // rows of R: conj(inner products) over the pivot norms
  for (int idx = tid; idx < N * k; idx += nt) Z[idx] = Q::conj_scale(Z[idx], bk.rinv<S>()[idx / N]);
  __syncthreads();
  *tail2 = t2;
  return k;
}

// Unpivoted Gram-Schmidt QR of Z (M x K, M >= K, column-major ld M), in place:
// on return column i of Z is 1 / bk.rinv()[i] times the i-th column of Q and R2
// (K x K, ld K) holds R.  Like pivoted_qr without the search.  Q is not used
// as an orthogonal matrix: Z V = Q (R2 V) holds to rounding whatever its
// orthogonality, and R2 is backward stable.
template <typename T>
__device__ void plain_qr(typename QA<T>::E* Z, int M, int K, typename QA<T>::E* R2, const QrBook& bk) {
  typedef QA<T> Q;
  typedef typename Q::E E;
  typedef typename Q::S S;
  S *rinv = bk.rinv<S>(), *n2 = bk.n2<S>(0);
  const int tid = threadIdx.x, nt = blockDim.x, lane32 = tid & 31;
  for (int j = tid >> 5; j < K; j += nt >> 5) {
    S acc = Q::zero();
    for (int r = lane32; r < M; r += 32) acc = Q::abs2_acc(Z[(size_t)j * M + r], acc);
    acc = Q::fin(Q::template group_sum<32>(acc));
    if (lane32 == 0) n2[j] = acc;
  }
  for (int idx = tid; idx < K * K; idx += nt) R2[idx] = Q::zeroE();
  __syncthreads();
  if constexpr (!Q::kFF) {
    float* key = bk.key(0);
    short* list = bk.list(0);
    for (int j = tid; j < K; j += nt) {
      key[j] = (float)n2[j];
      list[j] = (short)j;
    }
    __syncthreads();
    for (int i = 0; i < K; ++i) {
      GsStep g;
      g.X = Z;
      g.v = Z + (size_t)i * M;
      g.out = R2 + i;
      g.ostride = K;
      g.diag = g.out + (size_t)i * K;
      g.rinv = rinv + i;
      g.beta_sh = n2;
      g.key = key + i + 1;
      g.nkey = key + i + 1;
      g.list = list + i + 1;
      g.nlist = list + i + 1;
      g.R = M;
      g.nrest = K - i - 1;
      g.pos = INT_MAX;
      g.v2 = key[i];
      gs_step(g);
    }
  } else {
    for (int i = 0; i < K; ++i) {
      const S np = n2[i];
      const S ri = Q::rsqrt(np);
      const S beta = Q::mul(ri, ri);
      if (tid == 0) {
        rinv[i] = ri;
        R2[(size_t)i * K + i] = Q::realE(np);
      }
      const E* v = Z + (size_t)i * M;
      const int nrest = K - i - 1;
      const int G = qr_group(M, nrest);
      const int gl = tid & (G - 1), group = tid / G, ngroups = nt / G;
      for (int tb = 0; tb < nrest; tb += ngroups) {
        if (tb + (tid >> 5) * 32 / G >= nrest) break;
        const int t = tb + group;
        const bool act = t < nrest;
        E* cj = Z + (size_t)(act ? i + 1 + t : i) * M;
        S wr, wi, s2;
        const int j = act ? i + 1 + t : i;
        const float rb = inverse_bound(Q::tof(np), Q::tof(n2[j]));
        project<T>(v, cj, M, G, gl, act, beta, rb, wr, wi, s2);
        if (act && gl == 0) n2[j] = s2;
        if (act && gl == 0) {
          E z;
          z.x = wr;
          z.y = wi;
          R2[(size_t)(i + 1 + t) * K + i] = z;
        }
      }
      __syncthreads();
    }
  }
  for (int idx = tid; idx < K * K; idx += nt) R2[idx] = Q::scaleE(R2[idx], rinv[idx % K]);
  __syncthreads();
}

// Sweeps, with an FP64 finish for a double-float matrix whose double-float
// sweeps did not settle (converted in place -- both elements are 16 bytes --
// swept, converted back).  Leaves the FP64 column norms times `scale` in
// norm[] and the sweep counts in sh; returns the FP64 sweeps.
template <typename T>
__device__ int jacobi_norms(typename QA<T>::E* W, int m, int n, int ld, double scale, double* norm, JacobiShared* sh) {
  typedef QA<T> Q;
  typedef typename Q::S S;
  const int tid = threadIdx.x, nt = blockDim.x;
  int sw = jacobi_sweeps<T>(W, m, n, ld, reinterpret_cast<S*>(norm), sh);
  int sw64 = Q::kFF ? 0 : sw;
  bool settled = sw < JACOBI_MAX_SWEEPS;
  if (Q::kFF && !(settled || sh->noise_converged)) {
    cx<double>* Wd = reinterpret_cast<cx<double>*>(W);
    for (int j = 0; j < n; ++j)
      for (int r = tid; r < m; r += nt) Wd[(size_t)j * ld + r] = Q::to(W[(size_t)j * ld + r]);
    __syncthreads();
    sw64 = jacobi_sweeps<double>(Wd, m, n, ld, norm, sh);
    for (int j = 0; j < n; ++j)
      for (int r = tid; r < m; r += nt) W[(size_t)j * ld + r] = Q::from(Wd[(size_t)j * ld + r]);
    __syncthreads();
    settled = false;
  }
  if (!settled) {   // the sweeps' squared norms are not those of the result
    const int lane32 = tid & 31;
    for (int j = tid >> 5; j < n; j += nt >> 5) {
      S acc = Q::zero();
      for (int r = lane32; r < m; r += 32) acc = Q::abs2_acc(W[(size_t)j * ld + r], acc);
      acc = Q::fin(Q::template group_sum<32>(acc));
      if (lane32 == 0) reinterpret_cast<S*>(norm)[j] = acc;
    }
    __syncthreads();
  }
  for (int j = tid; j < n; j += nt) {
    const double n2 = Q::tod(reinterpret_cast<S*>(norm)[j]);
    norm[j] = n2 < 0.0 ? 0.0 : scale * sqrt(n2);   // NaN stays NaN
  }
  if (tid == 0) sh->sweeps32 = Q::kFF ? sw : 0;
  __syncthreads();
  return sw64;
}

// The split driver on X (R x N, ld R, the oriented matrix over `scale`, a
// power of two; destroyed), with Zg (R x N elements; FP64: and Mg, 2 N^2) as spare global storage,
// zs / zs_bytes spare shared memory and bkg spare global bookkeeping of
// qr_book_bytes(N).  x_shared says whether X itself is in shared memory.
// delta <= 0 selects the default cut.  Returns the kept rank; *Wout holds
// V_A Sigma (in the units of A / scale; N x k, ld N) with book->norm (in the
// units of A) / book->perm describing its columns in descending order.
template <typename T>
__device__ int qr_jacobi_truncate(typename QA<T>::E* X, bool x_shared, int R, int N, double scale,
                                  typename QA<T>::E* Zg, typename QA<T>::E* Mg, unsigned char* zs,
                                  size_t zs_bytes, unsigned char* bkg, double epsrel, float delta, SplitBook* book,
                                  JacobiShared* sh, typename QA<T>::E** Wout) {
  typedef QA<T> Q;
  typedef typename Q::E E;
  typedef typename Q::S S;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (!(delta > 0.f)) delta = qr_default_delta(Q::kFF, epsrel);
  double* norm = book->norm;
  int* perm = book->perm;
  QrBook bk;
  bk.N = N;
  bk.p = reinterpret_cast<unsigned char*>(book);
  if (qr_book_bytes(N) > sizeof(SplitBook)) {   // more than 383 columns
    if (qr_book_bytes(N) <= zs_bytes) {
      bk.p = zs;
      zs += (qr_book_bytes(N) + 15) & ~(size_t)15;
      zs_bytes -= (qr_book_bytes(N) + 15) & ~(size_t)15;
    } else {
      bk.p = bkg;
    }
  }
  // (the inverse pivot norms at bytes 16 N .. 24 N outlive the sweeps, which
  // use norm[0, k), and the ranking, which uses perm)
  // Z in shared memory when all N columns fit; the kept k may fit later
  E* Z = ((size_t)N * N * sizeof(E) <= zs_bytes) ? reinterpret_cast<E*>(zs) : Zg;
  float tail2;
  const int k = pivoted_qr<T>(X, R, N, delta, bk, Z, &tail2);
  const bool second = k >= 8 && 2 * k <= N;
  if (Z == Zg) {
    E* to = (size_t)N * k * sizeof(E) <= zs_bytes ? reinterpret_cast<E*>(zs) : (x_shared && !second ? X : Zg);
    if (to != Z) {
      for (int idx = tid; idx < N * k; idx += nt) to[idx] = Z[idx];
      Z = to;
      __syncthreads();
    }
  }
  if (second) {
    // Second QR, Z = Q2 R2: the Jacobi runs on the k x k R2 instead of the N
    // rows of Z (same singular values), and W = Q2 (R2 V) is formed for the
    // kept columns only, in sorted order.  X's storage: R2 and, behind it,
    // the kept columns: k^2 + N k <= R N for 2 k <= N <= R.
    E* R2 = X;
    E* Y = X + (size_t)k * k;
    S* rinv = bk.rinv<S>();
    plain_qr<T>(Z, N, k, R2, bk);
    if constexpr (!Q::kFF) {
      if (k >= PRESWEEP_MIN_COLS) {   // 4 k^2 <= R N
        E* W2 = presweep(R2, k, k, R2 + (size_t)k * k, R2 + (size_t)2 * k * k, reinterpret_cast<float*>(norm));
        if (W2 != R2) {
          for (int idx = tid; idx < k * k; idx += nt) R2[idx] = W2[idx];
          __syncthreads();
        }
      }
    }
    const int sw64 = jacobi_norms<T>(R2, k, k, k, scale, norm, sh);
    const int kk = jacobi_rank(k, epsrel, norm, perm, sh, sw64, tail2, scale);
    for (int idx = tid; idx < k * kk; idx += nt) {
      const int j = idx / k, i = idx - j * k;
      E* e = R2 + (size_t)perm[j] * k + i;
      *e = Q::scaleE(*e, rinv[i]);
    }
    __syncthreads();
    for (int idx = tid; idx < N * kk; idx += nt) {
      const int j = idx / N, r = idx - j * N;
      const E* y = R2 + (size_t)perm[j] * k;
      typename Q::Acc acc = Q::acc_zero();
#pragma unroll 4
      for (int i = 0; i < k; ++i) Q::acc_fma(acc, Z[(size_t)i * N + r], y[i]);
      Y[idx] = Q::acc_value(acc);
    }
    // the kept columns are stored sorted: norms in that order, identity perm
    for (int j = tid; j < kk; j += nt) norm[k + j] = norm[perm[j]];   // 2 k <= N
    __syncthreads();
    for (int j = tid; j < kk; j += nt) {
      norm[j] = norm[k + j];
      perm[j] = j;
    }
    __syncthreads();
    *Wout = Y;
    return kk;
  }
  if constexpr (!Q::kFF) {
    if (k >= PRESWEEP_MIN_COLS) {
      // scratch in X's storage (behind Z, when Z moved there) where it fits,
      // else in spare shared or global memory
      const size_t xfree = (size_t)R * N;
      size_t off = Z == X ? (size_t)N * k : 0;
      E* tmp = Zg;   // Z is in X: its global home is free
      if (off + (size_t)N * k <= xfree) {
        tmp = X + off;
        off += (size_t)N * k;
      }
      E* mats = Mg;
      if (off + presweep_mats(k) <= xfree)
        mats = X + off;
      else if (reinterpret_cast<unsigned char*>(Z) == zs &&
               ((size_t)N * k + presweep_mats(k)) * sizeof(E) <= zs_bytes)
        mats = reinterpret_cast<E*>(zs) + (size_t)N * k;
      Z = presweep(Z, N, k, tmp, mats, reinterpret_cast<float*>(norm));
    }
  }
  const int sw64 = jacobi_norms<T>(Z, N, k, N, scale, norm, sh);
  const int kk = jacobi_rank(k, epsrel, norm, perm, sh, sw64, tail2, scale);
  *Wout = Z;
  return kk;
}

}  // namespace otb
