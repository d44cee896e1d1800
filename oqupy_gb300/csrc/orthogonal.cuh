// Near-orthogonalisation of a complex128 split's Jacobi operand by matrix
// products: FP32 sweeps, the re-orthonormalised rotation applied in FP64 and
// first-order corrections, so that the FP64 sweeps that follow find almost
// nothing left to rotate.
//
// An FP64 instruction takes 64 clocks of an SM sub-partition, so an FP64 Jacobi
// round (5000 to 18000 clocks) is bound by that pipe, and an operand of k
// columns takes four to five sweeps of k rounds, 8 FP64 multiply-adds an
// element each.  All but the last digits of those rotations can be found in
// FP32, where a round takes 700 to 2000 clocks, and the products that replace
// the rest need 4 + 2 + 2 multiply-adds an element and column in all:
//   1. FP32 sweeps on a copy of Z; the same rotations on an identity give V,
//      unitary to ~1e-6;
//   2. E = V^H V - I in FP64, V <- V (I - E / 2 + 3 E^2 / 8): unitary to
//      rounding (the correction is 1e-6, double-float is enough for it);
//   3. W = Z V in FP64: columns orthogonal to ~1e-6;
//   4. PRESWEEP_CORRECTIONS times: Gram matrix of W in FP64, the small tangents
//      M of all pairs at once (antihermitian), W <- W (I + M + M^2 / 2), the
//      correction in double-float, then in FP32.  Unitary to |M|^3; pairs of
//      near-equal columns, whose angle is not small, are left out (M = 0).
// Every factor is unitary to rounding, so Z's singular values and the
// orthogonality that the sweeps then establish are what they are without this
// step; where the FP32 sweeps find nothing (NaN, zero columns) V is the
// identity.  The first correction leaves cosines of ~1e-12, the second ~1e-16
// (the sweeps rotate above 5e-16).
//
// Clocks of the whole orthogonalisation (256 threads), sweeps alone -> with
// this step: 12 x 8 171k -> 65k, 22 x 16 411k -> 147k, 37 x 28 1339k -> 486k,
// 60 x 44 3915k -> 1519k.  48 spin-boson instances at epsrel 1e-10: 12 steps in
// 243 instead of 362 ms.
#pragma once

#include "jacobi.cuh"

namespace otb {

// Splits of fewer columns go straight to the sweeps.  Sweeps keep a small column to
// its own rounding, products only to that of the largest one; but the QR's
// backward error is that of the largest one already, so a split is as accurate
// either way: singular values and the reconstruction to 4 N^1.5 unit roundoffs of
// the largest singular value (tests/test_split_numerics_gpu.py; exactly tied pairs
// over 0 to 9 decades, 8 to 40 columns, 12 operands each: singular values off by
// at most 9 unit roundoffs with products and 10 with sweeps, the smallest pair by
// the same 0.2 to 0.5, the reconstruction by at most 15 and 16).  What differs is
// which vector of a tied pair a truncation at that level keeps.  From 8 columns on
// the products are faster (three builds of 14 steps: 18.2 ms, 19.3 ms with 10, 22.2
// with 16); 10 is where the kept vectors of the narrow splits of a mean-field
// model with such a pair stay those of the sweeps (distance of its states from the
// reference at step 13: 6e-11 with 10, 12, 16 or no products, 1.1e-10 with 8).
// Double-float splits never take this way: their products run on the pipe that
// the sweeps are bound by (95 instances, splits of ~77 x 35: the 12 steps take
// 196 instead of 174 ms).
constexpr int PRESWEEP_MIN_COLS = 10;
constexpr int PRESWEEP_CORRECTIONS = 2;
constexpr float PRESWEEP_MIN_NORM2 = 1e-33f;   // B / A stays below 1e37 for norms of up to 1152 columns
constexpr float PRESWEEP_MAX_TAN = 4e-6f;   // larger tangents are left to the sweeps

// FP32 one-sided Jacobi sweeps on F (m + k rows, k columns, ld m + k): the
// inner products run over the first m rows, the rotations over all (the last k
// rows start as the identity and become V).  Same schedule and rotation as
// jacobi_sweeps.  Stops after a sweep whose largest cosine was below 1e-3: it
// leaves cosines of about the square, which the corrections finish.  RC rows a
// lane in registers (all of them with ALL), so that a round is one chain of
// load, product, reduction, angle and store: 28 columns of 37 + 28 rows take
// 1080 clocks a round, 1150 with the lower rows loaded after the rotation.
template <int G, int RC, bool ALL>
__device__ void presweeps32_rc(cx<float>* F, int m, int k, float* nrm2) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane32 = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int lane = tid & (G - 1), group = tid / G, ngroups = nt / G;
  const int np = (k + 1) >> 1, nr = (np << 1) - 1;
  const int ld = m + k;
  const float tol = 2.4e-7f, tol2 = tol * tol * (float)m;
  const bool up = lane & (G >> 1);
  for (int sweep = 0; sweep < 10; ++sweep) {
    for (int j = warp; j < k; j += nw) {
      float acc = 0.f;
      const cx<float>* c = F + (size_t)j * ld;
      for (int r = lane32; r < m; r += 32) acc = fmaf(c[r].x, c[r].x, fmaf(c[r].y, c[r].y, acc));
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (lane32 == 0) nrm2[j] = acc;
    }
    __syncthreads();
    bool large = false;
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
        const bool active = (p < np) && (b < k);
        cx<float>* ca = F + (size_t)(active ? a : 0) * ld;
        cx<float>* cb = F + (size_t)(active ? b : 0) * ld;
        const float A = nrm2[active ? a : 0], B = nrm2[active ? b : 0];
        cx<float> u[RC], v[RC];
        float gr = 0.f, gi = 0.f;
        for (int r0 = lane; r0 < (ALL ? lane + 1 : m); r0 += RC * G) {
#pragma unroll
          for (int q = 0; q < RC; ++q) {
            const int r = r0 + q * G;
            const bool in = active && r < (ALL ? ld : m);
            u[q] = in ? ca[r] : mk<float>(0.f, 0.f);
            v[q] = in ? cb[r] : mk<float>(0.f, 0.f);
          }
#pragma unroll
          for (int q = 0; q < RC; ++q)
            if (r0 + q * G < m) {
              gr = fmaf(u[q].x, v[q].x, fmaf(u[q].y, v[q].y, gr));
              gi = fmaf(u[q].x, v[q].y, fmaf(-u[q].y, v[q].x, gi));
            }
        }
        // gr in the group's lower half, gi in its upper half, then swapped
        float s = (up ? gi : gr) + __shfl_xor_sync(0xffffffffu, up ? gr : gi, G >> 1, 32);
#pragma unroll
        for (int off = G >> 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off, 32);
        const float o = __shfl_xor_sync(0xffffffffu, s, G >> 1, 32);
        const float rr = rsqrt_est(A) * rsqrt_est(B);
        const float x = (up ? o : s) * rr, y = (up ? s : o) * rr;
        const float c2 = fmaf(x, x, y * y);
        // columns at the end of FP32's range are left to the FP64 sweeps: above it
        // all of the angle's factors are finite (c2 is NaN for zero columns)
        if (active && c2 > tol2 && c2 < 1e30f && fminf(A, B) > PRESWEEP_MIN_NORM2) {
          large |= c2 > 1e-6f;
          const float d = 0.5f * ((B - A) * rr);
          const float hh = fmaf(d, d, c2);
          float q0 = rcp_est(fabsf(d) + hh * rsqrt_est(hh));
          q0 = d < 0.f ? -q0 : q0;
          const float tx = x * q0, ty = y * q0;
          const float w = fmaf(tx, tx, fmaf(ty, ty, 1.f)), e = rsqrt_est(w);
          const float c = e * fmaf(-0.5f * w * e, e, 1.5f);
          for (int r0 = lane; r0 < (ALL ? lane + 1 : ld); r0 += RC * G) {
            if (!ALL) {
#pragma unroll
              for (int q = 0; q < RC; ++q) {
                const int r = r0 + q * G;
                u[q] = r < ld ? ca[r] : mk<float>(0.f, 0.f);
                v[q] = r < ld ? cb[r] : mk<float>(0.f, 0.f);
              }
            }
#pragma unroll
            for (int q = 0; q < RC; ++q) {
              const cx<float> uu = u[q], vv = v[q];
              u[q].x = c * fmaf(-tx, vv.x, fmaf(-ty, vv.y, uu.x));
              u[q].y = c * fmaf(-tx, vv.y, fmaf(ty, vv.x, uu.y));
              v[q].x = c * fmaf(tx, uu.x, fmaf(-ty, uu.y, vv.x));
              v[q].y = c * fmaf(tx, uu.y, fmaf(ty, uu.x, vv.y));
            }
#pragma unroll
            for (int q = 0; q < RC; ++q) {
              const int r = r0 + q * G;
              if (r < ld) {
                ca[r] = u[q];
                cb[r] = v[q];
              }
            }
          }
          if (lane == 0) {
            const float tg = fmaf(tx, x, ty * y) * rcp_est(rr);   // tan(theta) |gamma|
            nrm2[a] = A - tg;
            nrm2[b] = B + tg;
          }
        }
      }
      if (round < nr - 1) __syncthreads();
    }
    if (!__syncthreads_or(large)) break;
  }
}

__device__ inline void presweeps32(cx<float>* F, int m, int k, float* nrm2) {
  const int rows = (m + k + 15) / 16;
  if (rows <= 3)
    presweeps32_rc<16, 3, true>(F, m, k, nrm2);
  else if (rows <= 5)
    presweeps32_rc<16, 5, true>(F, m, k, nrm2);
  else if (rows <= 8)
    presweeps32_rc<16, 8, true>(F, m, k, nrm2);
  else if (rows <= 12)
    presweeps32_rc<16, 12, true>(F, m, k, nrm2);
  else
    presweeps32_rc<32, 8, false>(F, m, k, nrm2);
}

// Elements of 16 bytes that presweep() needs beside Z and `tmp` (m k).
__host__ __device__ constexpr size_t presweep_mats(int k) { return (size_t)2 * k * k; }

// Upper-triangular index pairs of a k x k matrix (i <= j), folded so that every
// thread has work: t in [0, ((k + 1) / 2) (k + 1)).
__device__ __forceinline__ void fold_pair(int t, int k, int& i, int& j) {
  const int c = t / (k + 1), r = t - c * (k + 1);
  if (r <= c) {
    i = r;
    j = c;
  } else {
    i = r - c - 1;
    j = k - 1 - c;
  }
}

// sum_l a[l lda] b[l] over k terms in FP32.
__device__ __forceinline__ cx<float> product32(const cx<float>* a, int lda, const cx<float>* b, int k) {
  float sx = 0.f, sy = 0.f;
#pragma unroll 4
  for (int l = 0; l < k; ++l) {
    const cx<float> x = a[(size_t)l * lda], y = b[l];
    sx = fmaf(x.x, y.x, fmaf(-x.y, y.y, sx));
    sy = fmaf(x.x, y.y, fmaf(x.y, y.x, sy));
  }
  return mk<float>(sx, sy);
}

// FP64 -> double-float by integer instructions (trunc32).
__device__ __forceinline__ ff split32(double d) {
  unsigned rest;
  const float h = trunc32(d, &rest);
  // rest 2^(e - 52), e the exponent of d: FP32 2^e has h's exponent bits
  const float p = __uint_as_float(__float_as_uint(h) & 0xff800000u);   // +- 2^e
  const float l = __uint2float_rn(rest) * 2.220446049250313e-16f * p;
  const ff s = fast_two_sum(h, l);
  return s;
}
__device__ __forceinline__ cff split32(const cx<double>& a) {
  cff r;
  r.x = split32(a.x);
  r.y = split32(a.y);
  return r;
}

// Z (m x k, ld m, m >= k) -> W with nearly orthogonal columns, W = Z V with V
// unitary, in Z's or tmp's storage (returned).  work32 is the sweeps' workspace
// (k floats, shared).
__device__ inline cx<double>* presweep(cx<double>* Z, int m, int k, cx<double>* tmp, cx<double>* mats,
                                       float* work32) {
  typedef cx<double> E;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int ld = m + k;
  cx<float>* F = reinterpret_cast<cx<float>*>(tmp);   // (m + k) x k of 8 bytes <= m k of 16
  E* V = mats;
  for (int idx = tid; idx < ld * k; idx += nt) {
    const int j = idx / ld, r = idx - j * ld;
    F[idx] = r < m ? trunc32(Z[(size_t)j * m + r]) : mk<float>(r - m == j ? 1.f : 0.f, 0.f);
  }
  __syncthreads();
  presweeps32(F, m, k, work32);
  for (int idx = tid; idx < k * k; idx += nt) {
    const int j = idx / k, r = idx - j * k;
    const cx<float> v = F[(size_t)j * ld + m + r];
    V[idx] = mk<double>((double)v.x, (double)v.y);   // exact
  }
  __syncthreads();
  // F's storage: 1024 E and V in FP32; E, then C, in the second matrix
  cx<float>* Ef = reinterpret_cast<cx<float>*>(tmp);
  cx<float>* Vf = Ef + (size_t)k * k;
  E* Em = mats + (size_t)k * k;
  cff* C = reinterpret_cast<cff*>(Em);
  const int folds = ((k + 1) / 2) * (k + 1);
  for (int idx = tid; idx < k * k; idx += nt) Vf[idx] = trunc32(V[idx]);
  for (int t = tid; t < folds; t += nt) {   // E = V^H V - I
    int i, j;
    fold_pair(t, k, i, j);
    const E *a = V + (size_t)i * k, *b = V + (size_t)j * k;
    E e = mk<double>(i == j ? -1.0 : 0.0, 0.0);
#pragma unroll 4
    for (int l = 0; l < k; ++l) cjfma(e, a[l], b[l]);
    const cx<float> ef = mk<float>((float)(1024.0 * e.x), (float)(1024.0 * e.y));
    Em[(size_t)j * k + i] = e;
    Ef[(size_t)j * k + i] = ef;
    if (i != j) {
      Em[(size_t)i * k + j] = cconj(e);
      Ef[(size_t)i * k + j] = mk<float>(ef.x, -ef.y);
    }
  }
  __syncthreads();
  for (int idx = tid; idx < k * k; idx += nt) {   // C = -E / 2 + 3 E^2 / 8, in E's place
    const int j = idx / k, i = idx - j * k;
    const cx<float> sq = product32(Ef + i, k, Ef + (size_t)j * k, k);
    cff e = cff_scale(cff_from(Em[idx]), ff_make(-0.5f, 0.f));
    const float q = 0.375f / (1024.f * 1024.f);
    e.x = ff_add(e.x, ff_make(q * sq.x, 0.f));
    e.y = ff_add(e.y, ff_make(q * sq.y, 0.f));
    C[idx] = e;
  }
  __syncthreads();
  for (int idx = tid; idx < k * k; idx += nt) {   // V (I + C): the 1e-6 correction in double-float
    const int j = idx / k, r = idx - j * k;
    ccacc f = ccacc_zero();
#pragma unroll 2
    for (int l = 0; l < k; ++l) {
      const cx<float> v = Vf[(size_t)l * k + r];
      cff x;
      x.x = ff_make(v.x, 0.f);
      x.y = ff_make(v.y, 0.f);
      ccacc_fma(f, x, C[(size_t)j * k + l]);
    }
    V[idx] = V[idx] + ccacc_value(f);
  }
  __syncthreads();
  E* W = tmp;
  E* other = Z;
  for (int idx = tid; idx < m * k; idx += nt) {   // W = Z V
    const int j = idx / m, r = idx - j * m;
    E f = mk<double>(0.0, 0.0);
#pragma unroll 4
    for (int l = 0; l < k; ++l) cfma(f, Z[(size_t)l * m + r], V[(size_t)j * k + l]);
    W[idx] = f;
  }
  __syncthreads();
  cx<float>* M = reinterpret_cast<cx<float>*>(mats);   // tangents, k x k
  E* G = mats + (size_t)k * k;                         // Gram matrix, then
  cff* H = reinterpret_cast<cff*>(G);                  // M + M^2 / 2
#pragma unroll 1
  for (int pass = 0; pass < PRESWEEP_CORRECTIONS; ++pass) {
    for (int t = tid; t < folds; t += nt) {
      int i, j;
      fold_pair(t, k, i, j);
      const E *a = W + (size_t)i * m, *b = W + (size_t)j * m;
      E f = mk<double>(0.0, 0.0);
#pragma unroll 4
      for (int l = 0; l < m; ++l) cjfma(f, a[l], b[l]);
      G[(size_t)j * k + i] = f;
    }
    __syncthreads();
    for (int t = tid; t < folds; t += nt) {
      int i, j;
      fold_pair(t, k, i, j);
      cx<float> t2 = mk<float>(0.f, 0.f);
      if (i < j) {
        const double ga = G[(size_t)i * k + i].x, gb = G[(size_t)j * k + j].x;
        const float rr = rsqrt_est((float)ga) * rsqrt_est((float)gb);
        const E g = G[(size_t)j * k + i];
        const float x = (float)(g.x * (double)rr), y = (float)(g.y * (double)rr);
        const float c2 = fmaf(x, x, y * y);
        const float d = 0.5f * ((float)(gb - ga) * rr);
        const float hh = fmaf(d, d, c2);
        float q = rcp_est(fabsf(d) + hh * rsqrt_est(hh));
        q = d < 0.f ? -q : q;
        // false for NaN (zero columns, zero cosines) and for pairs of near-equal columns
        if (c2 * q * q <= PRESWEEP_MAX_TAN * PRESWEEP_MAX_TAN) t2 = mk<float>(x * q, y * q);
        M[(size_t)i * k + j] = mk<float>(-t2.x, t2.y);
      }
      M[(size_t)j * k + i] = t2;
    }
    __syncthreads();
    for (int idx = tid; idx < k * k; idx += nt) {
      const int j = idx / k, i = idx - j * k;
      const cx<float> sq = product32(M + i, k, M + (size_t)j * k, k);
      cff h;
      h.x = two_sum(M[idx].x, 0.5f * sq.x);
      h.y = two_sum(M[idx].y, 0.5f * sq.y);
      H[idx] = h;
    }
    __syncthreads();
    // W (I + H): the first pass's correction (1e-6) in double-float, the
    // second's (1e-12) in FP32
    for (int idx = tid; idx < m * k; idx += nt) {
      const int j = idx / m, r = idx - j * m;
      E e;
      if (pass > 0) {
        float sx = 0.f, sy = 0.f;
#pragma unroll 4
        for (int l = 0; l < k; ++l) {
          const cx<float> x = trunc32(W[(size_t)l * m + r]);
          const cff y = H[(size_t)j * k + l];
          sx = fmaf(x.x, y.x.hi, fmaf(-x.y, y.y.hi, sx));
          sy = fmaf(x.x, y.y.hi, fmaf(x.y, y.x.hi, sy));
        }
        e = mk<double>((double)sx, (double)sy);
      } else {
        ccacc f = ccacc_zero();
#pragma unroll 2
        for (int l = 0; l < k; ++l) ccacc_fma(f, split32(W[(size_t)l * m + r]), H[(size_t)j * k + l]);
        e = ccacc_value(f);
      }
      other[idx] = W[idx] + e;
    }
    __syncthreads();
    E* const s = W;
    W = other;
    other = s;
  }
  return W;
}

}  // namespace otb
