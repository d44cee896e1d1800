// One-sided (Hestenes) Jacobi SVD with the TEMPO relative truncation rule,
// executed by one CTA on a matrix held in shared or global memory.
//
// Replaces, for every bond split on the TEMPO / PT-TEMPO path, the
// truncated SVD the reference obtains from tensornetwork's
// split_node_full_svd(max_truncation_err=epsrel, relative=True)
// (oqupy/backends/node_array.py:262-268, 285-291, 541-547).  The truncation
// rule keeps chi = #{i : sqrt(sum_{j>=i} s_j^2) > epsrel * s_0} over the
// singular values in descending order (stated in the reference at
// oqupy/mps_mpo.py:452-457).
//
// Arithmetic (template parameter T): double (complex128 form) or ff
// (double-float on the FP32 pipe, the mixed form).  The rank decision is
// always FP64.
#pragma once

#include "arith.cuh"

namespace otb {

constexpr int JACOBI_MAX_SWEEPS = 60;

struct JacobiShared {
  unsigned worst;   // largest relative off-diagonal rotated in the last allowed sweep (float bits)
  unsigned c2max[2], t2max[2];   // largest rotated squared cosine and scaled tangent of a sweep (float bits)
  int noise_converged;
  int kept;
  int status;
  int sweeps;     // FP64 sweeps of the last split
  int sweeps32;   // double-float sweeps of the last split (mixed form)
};

// Lanes per column pair: 16, so that small operands occupy the SM's four
// schedulers, and 8 from 17 pairs on.  Wider groups repeat the pair's scalar
// work (reduction and rotation parameters, ~170 instructions) in more warps and
// a round becomes issue-bound; narrower ones leave schedulers idle while a warp
// issues its rows one after another.  Clocks per round on 8 / 16 / 32 lanes,
// double-float: 8 pairs 1511 / 1339 / 1435, 12 pairs 1784 / 1752 / 2313, 25
// pairs 4134 / 4443 / 5515; FP64: 10 pairs 5691 / 4969 / 8573, 18 pairs 11474 /
// 15223 / 17043.
__device__ __forceinline__ int jacobi_group(int pairs, int rows) { return (pairs <= 16 || rows > 128) ? 16 : 8; }

// Sweeps of one-sided Jacobi on W (m x n, column-major, leading dim ld).
// nrm2 holds n scalars of workspace in shared memory; when the sweeps settle
// (return value < JACOBI_MAX_SWEEPS) it holds the squared column norms of the
// result.  Returns the number of sweeps with a rotation.
//
// Parallel schedule: round-robin ("circle") tournament over the columns; the
// n/2 disjoint pairs of a round rotate concurrently, one __syncthreads per
// round.  A pair is owned by G lanes.
//
// What bounds it: the chain load -> inner product -> reduction -> angle ->
// rotation of one round, of which a split of ~20 columns has about 90 (small
// operands), the FP32 issue rate (large ones, double-float) or the FP64 pipe,
// where a warp instruction takes 64 clocks of its scheduler (complex128 form).
// Hence
//  * only the pair's inner product gamma is reduced (QA<T>::gamma).  The squared
//    norms are kept beside the matrix, recomputed at the start of every sweep
//    and updated by -+ tan(theta) |gamma| with each rotation (they only steer
//    the angle and the thresholds; a sweep without a rotation has exact ones);
//  * the complex tangent tau is formed in FP32 from hardware estimates: its
//    error only leaves a relative 1e-6 of gamma behind, which the next sweep
//    removes.  What has to hold to full precision is unitarity: tau is exact in
//    either arithmetic, and u - conj(tau) v, v + tau u are exactly orthogonal
//    combinations whose common scale c = 1 / sqrt(1 + |tau|^2) is formed while
//    they are.
// One round of a 22 x 16 double-float operand: 3700 (angle and phase in
// double-float, norms and gamma reduced by error-free additions) -> 1340
// clocks; a 27 x 20 FP64 one: 16100 -> 4970.
//
// The last sweep is known without another one to check it.  A rotation leaves
// 1e-6 of its pair's cosine (the FP32 angle), and changes the cosine of column u
// with any third column w by |tau| |v| / |u| cos(v, w); over the rest of the
// sweep a pair sees at most 2 n of these.  When the largest cosine rotated in a
// sweep times (2e-6 + 2 n times the largest |tau| |v| / |u|) is below half the
// rotation threshold, the next sweep would rotate nothing, and only the norms
// are formed anew.  253 double-float instances, 40 steps: 265 -> 260 ms; 48
// complex128 ones, 12 steps (two sweeps after the products' rotations, now
// mostly one): 221 -> 210 ms.
//
// Numerical-zero floor: a column whose squared norm is below (16 sqrt(m) eps)^2
// (double-float: (32 sqrt(m) eps)^2) times the largest squared column norm
// holds only rounding noise of the other columns; pairs involving such a
// column are not rotated (rotating noise against a real column regenerates
// noise at the stopping threshold and never converges).  The floor changes
// nothing above the rounding level of the decomposition.
// RC: rows a lane holds in registers at a time; with ALL they are all of its
// rows (m <= RC G), loaded once per pair, so that a row's loads never wait for
// another row's stores.
template <typename T, int G, int RC, bool ALL>
__device__ int jacobi_sweeps_rc(typename QA<T>::E* W, int m, int n, int ld, typename QA<T>::S* nrm2, JacobiShared* sh) {
  typedef QA<T> Q;
  typedef typename Q::E E;
  typedef typename Q::S S;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane32 = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int lane = tid & (G - 1);
  const int group = tid / G;
  const int ngroups = nt / G;
  const int np = (n + 1) >> 1;
  const int nr = (np << 1) - 1;   // rounds of a sweep
  const float tol = Q::jacobi_tol(m), zf = Q::jacobi_floor(m);
  const float tol2 = tol * tol;
  if (tid == 0) {
    sh->noise_converged = 0;
    sh->worst = 0u;
    sh->c2max[0] = sh->t2max[0] = 0u;
  }
  int sweep;
  bool done = false;
  for (sweep = 0; sweep < JACOBI_MAX_SWEEPS; ++sweep) {
    // squared column norms, and the largest (a lower bound of s_max^2)
    for (int j = warp; j < n; j += nw) {
      S acc = Q::zero();
      const E* c = W + (size_t)j * ld;
      for (int r = lane32; r < m; r += 32) acc = Q::abs2_acc(c[r], acc);
      acc = Q::template group_sum<32>(acc);
      if (lane32 == 0) nrm2[j] = Q::fin(acc);
    }
    __syncthreads();
    if (done) break;
    const int par = sweep & 1;
    if (tid == 0) sh->c2max[par ^ 1] = sh->t2max[par ^ 1] = 0u;
    float c2m = 0.f, t2m = 0.f;
    unsigned mxb = 0u;
    for (int j = lane32; j < n; j += 32) mxb = max(mxb, __float_as_uint(Q::tof(nrm2[j])));
    const float zfloor = zf * zf * __uint_as_float(__reduce_max_sync(0xffffffffu, mxb));
    bool rotated = false;
    for (int round = 0; round < nr; ++round) {
      for (int pb = 0; pb < np; pb += ngroups) {
        if (pb + (warp * 32) / G >= np) break;   // no pair left for this warp
        const int p = pb + group;
        int a, b;
        if (p == 0) {
          a = nr;
          b = round;
        } else {
          a = round + p;
          a = a >= nr ? a - nr : a;
          b = round - p;
          b = b < 0 ? b + nr : b;
        }
        if (a > b) {
          const int t = a;
          a = b;
          b = t;
        }
        const bool active = (p < np) && (b < n);
        E* ca = W + (size_t)(active ? a : 0) * ld;
        E* cb = W + (size_t)(active ? b : 0) * ld;
        const S na = nrm2[active ? a : 0], nb = nrm2[active ? b : 0];
        S gr = Q::zero(), gi = Q::zero();
        E u[RC], v[RC];
        for (int r0 = lane; r0 < (ALL ? lane + 1 : m); r0 += RC * G) {
#pragma unroll
          for (int q = 0; q < RC; ++q) {
            const bool in = active && r0 + q * G < m;
            u[q] = in ? ca[r0 + q * G] : Q::zeroE();
            v[q] = in ? cb[r0 + q * G] : Q::zeroE();
          }
#pragma unroll
          for (int q = 0; q < RC; ++q) Q::dotj(gr, gi, u[q], v[q]);
        }
        const float A = Q::tof(na), B = Q::tof(nb);
        const float rr = rsqrt_est(A) * rsqrt_est(B);
        float x, y;   // gamma / (|u| |v|)
        Q::template gamma<G>(gr, gi, rr, x, y);
        const float c2 = fmaf(x, x, y * y);
        if (active && A > zfloor && B > zfloor && c2 > tol2) {
          rotated = true;
          // tan(2 theta) = |gamma| / d, d = (B - A) / 2; tau = tan(theta) e^{i phi}
          const float d = 0.5f * (Q::diff(nb, na) * rr);
          const float hh = fmaf(d, d, c2);
          float q0 = rcp_est(fabsf(d) + hh * rsqrt_est(hh));
          q0 = d < 0.f ? -q0 : q0;
          const float tx = x * q0, ty = y * q0;
          const float ratio = fmaxf(A, B) * rr;
          c2m = fmaxf(c2m, c2);
          t2m = fmaxf(t2m, fmaf(tx, tx, ty * ty) * (ratio * ratio));
          const typename Q::Rot rot = Q::rotation(tx, ty);
          for (int r0 = lane; r0 < (ALL ? lane + 1 : m); r0 += RC * G) {
#pragma unroll
            for (int q = 0; q < RC; ++q) {
              if (!ALL) {
                const bool in = r0 + q * G < m;
                u[q] = in ? ca[r0 + q * G] : Q::zeroE();
                v[q] = in ? cb[r0 + q * G] : Q::zeroE();
              }
            }
#pragma unroll
            for (int q = 0; q < RC; ++q) Q::rotate(rot, u[q], v[q]);
#pragma unroll
            for (int q = 0; q < RC; ++q)
              if (r0 + q * G < m) {
                ca[r0 + q * G] = u[q];
                cb[r0 + q * G] = v[q];
              }
          }
          if (lane == 0) {
            const float tg = __fdividef(fmaf(tx, x, ty * y), rr);   // tan(theta) |gamma|
            nrm2[a] = Q::shift(na, -tg);
            nrm2[b] = Q::shift(nb, tg);
            if (sweep == JACOBI_MAX_SWEEPS - 1) atomicMax(&sh->worst, __float_as_uint(sqrtf(c2)));
          }
        }
      }
      if (round < nr - 1) __syncthreads();
    }
    {
      const unsigned cb = __reduce_max_sync(0xffffffffu, __float_as_uint(c2m));
      const unsigned tb = __reduce_max_sync(0xffffffffu, __float_as_uint(t2m));
      if (lane32 == 0 && cb) {
        atomicMax(&sh->c2max[par], cb);
        atomicMax(&sh->t2max[par], tb);
      }
    }
    if (!__syncthreads_or(rotated)) break;
    const float left = 2e-6f + 4.f * (float)np * sqrtf(__uint_as_float(sh->t2max[par]));
    done = __uint_as_float(sh->c2max[par]) * (left * left) < 0.25f * tol2;
  }
  // at the sweep cap, rotations below 1e-10 relative are rounding noise
  if (sweep == JACOBI_MAX_SWEEPS && tid == 0 && __uint_as_float(sh->worst) < 1e-10f) sh->noise_converged = 1;
  __syncthreads();   // publish noise_converged
  return sweep;
}

template <typename T>
__device__ int jacobi_sweeps(typename QA<T>::E* W, int m, int n, int ld, typename QA<T>::S* nrm2, JacobiShared* sh) {
  const int G = jacobi_group((n + 1) >> 1, m);
  const int rows = (m + G - 1) / G;
  if (G == 8) {
    if (rows <= 2) return jacobi_sweeps_rc<T, 8, 2, true>(W, m, n, ld, nrm2, sh);
    if (rows == 3) return jacobi_sweeps_rc<T, 8, 3, true>(W, m, n, ld, nrm2, sh);
    if (rows == 4) return jacobi_sweeps_rc<T, 8, 4, true>(W, m, n, ld, nrm2, sh);
    if (rows <= 6) return jacobi_sweeps_rc<T, 8, 3, false>(W, m, n, ld, nrm2, sh);
    return jacobi_sweeps_rc<T, 8, 4, false>(W, m, n, ld, nrm2, sh);
  }
  if (rows <= 2) return jacobi_sweeps_rc<T, 16, 2, true>(W, m, n, ld, nrm2, sh);
  if (rows == 3) return jacobi_sweeps_rc<T, 16, 3, true>(W, m, n, ld, nrm2, sh);
  if (rows == 4) return jacobi_sweeps_rc<T, 16, 4, true>(W, m, n, ld, nrm2, sh);
  return jacobi_sweeps_rc<T, 16, 4, false>(W, m, n, ld, nrm2, sh);
}

// Descending order of the n values norm[] and the kept rank (>= 1).  tail2 is the
// squared norm, over scale^2, of a block dropped before the sweeps.  Where the
// largest value is below 2^-400 or above 2^400, squares are summed in units of a
// power of two next to it, so that their sum stays in range; a largest value
// whose own square does not is refused.
__device__ inline int jacobi_rank(int n, double epsrel, double* norm, int* perm, JacobiShared* sh,
                                  int sweeps, double tail2, double scale) {
  const int tid = threadIdx.x;
  const int nthreads = blockDim.x;
  // norms are >= 0: their bit patterns order like the values (no FP64 compare)
  for (int j = tid; j < n; j += nthreads) {
    const long long sj = __double_as_longlong(norm[j]);
    int rank = 0;
    for (int i = 0; i < n; ++i) {
      const long long si = __double_as_longlong(norm[i]);
      rank += (si > sj) || (si == sj && i < j);
    }
    perm[rank] = j;
  }
  __syncthreads();
  if (tid == 0) {
    const double s0 = norm[perm[0]];
    const int e = (__double2hiint(s0) >> 20) & 0x7ff;
    double cum;
    int kept = 0;
    // (the units cost an FP64 multiplication a value: 1 % of small splits)
    if (e > 623 && e < 1423) {
      const double thr = epsrel * s0, thr2 = thr * thr;
      cum = tail2 * scale * scale;  // a block dropped before the sweeps is all in the tail
#pragma unroll 4
      for (int r = n - 1; r >= 0; --r) {
        const double s = norm[perm[r]];
        cum = fma(s, s, cum);
        kept += (cum > thr2) ? 1 : 0;
      }
    } else {
      const double unit = __hiloint2double((e > 1 && e < 2045 ? 2046 - e : 1023) << 20, 0);   // about 1 / s0
      const double thr = epsrel * (s0 * unit), thr2 = thr * thr;
      cum = tail2 * (scale * unit) * (scale * unit);
      for (int r = n - 1; r >= 0; --r) {
        const double s = norm[perm[r]] * unit;
        cum = fma(s, s, cum);
        kept += (cum > thr2) ? 1 : 0;
      }
      if (!isfinite(s0 * s0)) cum = s0 * s0;
    }
    if (kept < 1) kept = 1;
    sh->kept = kept;
    sh->sweeps = sweeps;
    sh->status = ST_OK;
    if (!isfinite(cum))
      sh->status = ST_NONFINITE;
    else if (sweeps >= JACOBI_MAX_SWEEPS && !sh->noise_converged)
      sh->status = ST_NO_CONVERGENCE;
  }
  __syncthreads();
  return sh->kept;
}

}  // namespace otb
