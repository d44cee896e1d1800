// Process-tensor sweep (compute_dynamics hot loop), batched over systems.
//
// Reference: compute_dynamics (oqupy/system_dynamics.py:131-165) with
// _apply_system_superoperator (:631-640), _apply_pt_mpos (:654-700) and
// _apply_caps (:643-651).  For a rank-3 PT-MPO tensor T_k[l][r][a] (delta
// between input and output legs, process_tensor.py:346-347) one step of
// system h is
//     u[l][a]  = sum_b P1_hk[a][b] v[l][b]
//     w[r][a]  = sum_l u[l][a] T_k[l][r][a]          (T_k = d * site_k[l][a][r])
//     v'[r][a] = sum_b P2_hk[a][b] w[r][b]
//     rho_h(k+1)[a] = sum_r v'[r][a] cap_{k+1}[r]
// (P1_hk, P2_hk) is entry pidx[h][k] of a table of propagator pairs: a
// time-dependent system has one pair per step, and control operations
// (system_dynamics.py:131-160) are folded into the pairs of their steps on
// the host -- a post-measurement control of step k into P1_hk (P1 post_k),
// a pre-measurement control of step k+1 into P2_hk (pre_{k+1} P2).  A
// transform_in / transform_out of the process tensor is folded into P1 / P2 on
// the host.  Whole sweeps run in one launch (sweep_kernel, below);
// dyn_step_kernel does one step at a time for callers that decide the next
// propagators from the states in between (grid: bond chunks x systems).  Both
// are reproducible bit for bit.  dyn_step_kernel's read-out: a CTA adds its
// bond chunk's terms in a fixed order, and the last CTA of a system to finish
// (counted after a memory fence) adds the chunks' partial sums in chunk order.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "engine.h"

namespace otb {

namespace cg = cooperative_groups;

typedef cx<double> zc;
constexpr int DYN_RB = 32;       // output bond indices per CTA
constexpr int DYN_THREADS = 128;

// Eight CTAs per SM (64 registers): left to itself the compiler takes 32 and
// spills.  A session of one system: 60 steps at bond 90 (D = 4) 2750 -> 2620 us,
// 2748 with 40 registers; 24 steps at bond 55 (D = 9) 1840 -> 1605 us; 1024 systems
// 14.8 -> 14.7 and 8.2 -> 8.1 ms.
__global__ void __launch_bounds__(DYN_THREADS, 8) dyn_step_kernel(DynLaunch L) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ int last;
  const int h = blockIdx.y;
  const int k = L.k;
  const int D = L.D;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int2 dm = L.dims[k];
  const int l = dm.x, r = dm.y;
  const zc* A = (const zc*)L.sites + (long long)k * L.slot_elems;
  zc* u = (zc*)dsm;
  zc* w = u + l * D;
  const zc* v = (const zc*)L.vcur + (long long)h * L.cap * D;
  const zc* P1 = (const zc*)L.ptab + (long long)L.pidx[(long long)h * L.pidx_stride + k] * 2 * D * D;
  const zc* P2 = P1 + D * D;
  for (int idx = tid; idx < l * D; idx += nt) {
    const int ll = idx / D, a = idx - ll * D;
    zc acc = mk<double>(0, 0);
    for (int b = 0; b < D; ++b) cfma(acc, P1[a * D + b], v[ll * D + b]);
    u[idx] = acc;
  }
  __syncthreads();
  const int r0 = blockIdx.x * DYN_RB;
  const int rn = min(DYN_RB, r - r0);
  for (int idx = tid; idx < rn * D; idx += nt) {
    const int a = idx / rn, rr = idx - a * rn;
    zc acc = mk<double>(0, 0);
    for (int ll = 0; ll < l; ++ll) cfma(acc, u[ll * D + a], A[((size_t)ll * D + a) * r + r0 + rr]);
    w[rr * D + a] = cscale(acc, (double)L.d);
  }
  __syncthreads();
  zc* vn = (zc*)L.vnext + (long long)h * L.cap * D;
  const zc* capn = (const zc*)L.caps + (long long)(k + 1) * L.cap;
  zc* cb = w + DYN_RB * D;   // read-out terms of this chunk, [rr][a]
  for (int idx = tid; idx < rn * D; idx += nt) {
    const int rr = idx / D, a = idx - rr * D;
    zc y = mk<double>(0, 0);
    for (int b = 0; b < D; ++b) cfma(y, P2[a * D + b], w[rr * D + b]);
    vn[(size_t)(r0 + rr) * D + a] = y;
    cb[idx] = cmul(y, capn[r0 + rr]);
  }
  __syncthreads();
  zc* part = (zc*)L.partial + (long long)h * L.max_chunks * D;
  if (tid < D) {
    zc acc = mk<double>(0, 0);
    for (int rr = 0; rr < rn; ++rr) acc = acc + cb[rr * D + tid];
    part[blockIdx.x * D + tid] = acc;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = (atomicAdd(L.counter + h, 1u) == gridDim.x - 1) ? 1 : 0;
  __syncthreads();
  if (last) {
    if (tid < D) {
      zc acc = mk<double>(0, 0);
      for (int c = 0; c < (int)gridDim.x; ++c) {
        const double2 q = __ldcg(reinterpret_cast<const double2*>(part + c * D + tid));
        acc = acc + mk<double>(q.x, q.y);
      }
      zc* out = (zc*)L.out + (long long)(k + 1) * L.nh * D + (long long)h * D;
      out[tid] = acc;
    }
    if (tid == 0) L.counter[h] = 0u;
  }
}

__global__ void dyn_init_kernel(DynLaunch L, const double* rho0) {
  // v_0 = rho0 (bond dimension 1); rho(0) = rho0 * cap_0[0]
  const int h = blockIdx.x;
  const int D = L.D;
  const zc* r0 = (const zc*)rho0 + (long long)h * D;
  zc* v = (zc*)L.vcur + (long long)h * L.cap * D;
  const zc c0 = ((const zc*)L.caps)[0];
  for (int a = threadIdx.x; a < D; a += blockDim.x) {
    v[a] = r0[a];
    const zc s = cmul(r0[a], c0);
    L.out[2 * ((long long)h * D + a)] = s.x;
    L.out[2 * ((long long)h * D + a) + 1] = s.y;
  }
}

// ---------------------------------------------------------------------------
// Whole sweeps: all steps of a system in one launch
// ---------------------------------------------------------------------------
//
// A system's steps depend on each other but on no other system, so a sweep of
// N steps is one kernel: a cluster of C CTAs (C = 1 for many systems) carries S
// systems through all steps and exchanges the new states through distributed
// shared memory, one cluster barrier per step.  With u_k = P1_k v_k a step is
//     w[r][a]      = sum_l u_k[l][a] A_k[l][a][r]
//     u_{k+1}[r]   = Q_k w[r],           Q_k  = d P1_{k+1} P2_k
//     rho_h(k+1)   = d P2_k y,           y[a] = sum_l u_k[l][a] B_k[l][a],
//     B_k[l][a]    = sum_r A_k[l][a][r] cap_{k+1}[r]
// (d P2_k w is the state with its bond leg).  B depends on the process tensor
// only and enters as one more column r of A_k, which makes the read-out part of
// the contraction instead of a reduction over r; Q saves one of the two
// propagator products per step.
//
// What bounds it: the FP64 pipe (a warp instruction takes 64 clocks of its
// scheduler): 4 l r D multiply-adds per step and system, and for few systems
// the step's chain of dependent phases.  Hence C splits the columns r of few
// systems over SMs, S lets many systems share every load of A, and a column's
// sum over l is split over G lanes where a CTA has fewer columns than threads.
// One launch replaces a graph of N kernel nodes that had to be captured and
// instantiated per call. Whole calls, 60 steps, bond 13, before and now: 8
// systems 760 and 240 us, 1024 systems 1750 and 920 us, gradient of 24 driven
// systems 1610 and 500 us.
constexpr int SWEEP_THREADS = 256;

__global__ void __launch_bounds__(SWEEP_THREADS) sweep_prepare_kernel(SweepLaunch L) {
  const int D = L.D;
  const int nt = gridDim.y * blockDim.x, t0 = blockIdx.y * blockDim.x + threadIdx.x;
  const int k = blockIdx.x;
  // B_k
  {
    const int2 dm = L.dims[k];
    const zc* A = (const zc*)L.sites + (long long)k * L.slot_elems;
    const zc* capn = (const zc*)L.caps + (long long)(k + 1) * L.cap;
    zc* B = (zc*)L.bcol + (long long)k * L.cap * D;
    // eight lanes per entry
    const int g = t0 & 7;
    for (int e0 = (t0 >> 3) & ~3; e0 < dm.x * D; e0 += nt >> 3) {   // warp-uniform trip count
      const int e = e0 + ((t0 >> 3) & 3);
      zc acc = mk<double>(0, 0);
      if (e < dm.x * D)
        for (int rr = g; rr < dm.y; rr += 8) cfma(acc, A[(size_t)e * dm.y + rr], capn[rr]);
      for (int off = 4; off > 0; off >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
      }
      if (g == 0 && e < dm.x * D) B[e] = acc;
    }
  }
  // Q_k and d P2_k of every system (of step 0 only when they do not change)
  if (k > 0 && !L.pidx) return;
  const double d = (double)L.d;
  for (int idx = t0; idx < L.nh * D * D; idx += nt) {
    const int h = idx / (D * D), e = idx - h * D * D;
    const int a = e / D, c = e - a * D;
    const int i0 = L.pidx ? L.pidx[(long long)h * L.num_steps + k] : h;
    const int i1 = L.pidx ? L.pidx[(long long)h * L.num_steps + min(k + 1, L.num_steps - 1)] : h;
    const zc* P2 = (const zc*)L.ptab + ((long long)i0 * 2 + 1) * D * D;
    const zc* P1n = (const zc*)L.ptab + (long long)i1 * 2 * D * D;
    zc acc = mk<double>(0, 0);
    for (int b = 0; b < D; ++b) cfma(acc, P1n[a * D + b], P2[b * D + c]);
    zc* Q = (zc*)L.qtab + ((long long)(L.pidx ? k : 0) * L.nh + h) * 2 * D * D;
    Q[e] = cscale(acc, d);
    Q[D * D + e] = cscale(P2[e], d);
  }
}

// 16-byte asynchronous copy global -> shared.
__device__ __forceinline__ void copy16(zc* dst, const zc* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void lane_sum(zc& v, int G) {
  for (int off = G >> 1; off > 0; off >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
  }
}

// A column's sum over `len` terms is split into V partial sums (terms v, v + V,
// ...; added by halves, as lane_sum adds lanes), whatever the number of systems
// and of CTAs that share a step, so that a system's states are the same bits in
// any batch.  V is the number of lanes a column gets where one CTA holds all
// `outs` columns of the step, and at least 4 for steps wide enough to be split
// over a cluster, whose CTAs have lanes left over (bonds from 20 on with D = 4);
// a CTA with too many columns for V lanes each adds the rest one after the
// other (WIDE kernels; without such a step every column has its V lanes).  The
// parts cost a wide sweep that has a CTA or more per SM up to 5 % (bond 85: 77
// systems 2115 -> 2225 us, 1024 systems 12.3 -> 12.5 ms; with G after the CTA's own
// columns, but other bits in every batch).
__host__ __device__ __forceinline__ int sum_parts(int len, int outs) {
  int V = 1;
  while (V < 8 && 4 * V <= len && (2 * V * outs <= SWEEP_THREADS || (V < 4 && len * outs > 1500))) V <<= 1;
  return V;
}
__host__ __device__ __forceinline__ int part_lanes(int V, int outs) {
  int G = 1;
  while (G < V && 2 * G * outs <= SWEEP_THREADS) G <<= 1;
  return G;
}
// The j-th part of V / G that lane g adds up, in the order in which halves are
// added: 0 2 1 3 of four.
__device__ __forceinline__ int part_index(int j, int g, int G, int parts) {
  return g + G * (parts == 4 ? ((j & 1) << 1) | (j >> 1) : j);
}
__device__ __forceinline__ void add_part(int j, const zc& part, zc& sum, zc& hold) {
  if (j == 0)
    sum = part;
  else if (j == 1)
    sum = sum + part;
  else if (j == 2)
    hold = part;
  else
    sum = sum + (hold + part);
}

// CTAs per SM that the register allocation aims at: one CTA's chain of phases is
// what counts (168 registers for four systems), but with one system's partial
// sums after each other the compiler's longer unrolling costs more than it hides
// (77 systems, bond 85: 2350 us a sweep without a bound, 2225 with).
__host__ __device__ constexpr int sweep_ctas(bool lean, int dt) { return !lean ? 1 : dt == 4 ? 3 : 2; }

// sum_a M[a ms] x[a] over D terms.
__device__ __forceinline__ zc row_product(const zc* M, int ms, const zc* x, int D) {
  zc acc = mk<double>(0, 0);
  for (int a = 0; a < D; ++a) cfma(acc, M[a * ms], x[a]);
  return acc;
}

// This CTA's columns of step k, into shared memory: to[(l D + a) nc + cc].
__device__ __forceinline__ void stage_columns(const SweepLaunch& L, int k, int2 dm, int c0, int nc, zc* to) {
  const int D = L.D, r = dm.y;
  const zc* A = (const zc*)L.sites + (long long)k * L.slot_elems + c0;
  const zc* B = (const zc*)L.bcol + (long long)k * L.cap * D;
  // one warp per row (no index division: the copies of a step take longer to
  // address than to make)
  for (int row = threadIdx.x >> 5; row < dm.x * D; row += SWEEP_THREADS / 32)
    for (int cc = threadIdx.x & 31; cc < nc; cc += 32)
      copy16(to + row * nc + cc, c0 + cc == r ? B + row : A + (size_t)row * r + cc);
}

// S systems per CTA; RECORD keeps v_k (gradient sweeps); DT as below.  With L.stage the next
// step's columns (and propagators) are copied to shared memory while a step
// computes: a step waits for no global load.
template <int S, bool RECORD, int DT, bool WIDE>
__global__ void __launch_bounds__(SWEEP_THREADS, sweep_ctas(WIDE && S == 1, DT)) sweep_kernel(SweepLaunch L) {
  extern __shared__ __align__(16) unsigned char dsm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), c = (int)cluster.block_rank();
  const int D = DT ? DT : L.D, DD = D * D;   // DT: the Liouville dimension, 0 = given at run time
  const int tid = threadIdx.x;
  constexpr int nt = SWEEP_THREADS;
  const int h0 = (int)(blockIdx.x / C) * S;
  const int ns = min(S, L.nh - h0);
  const int ustride = L.max_bond * D;               // one system's states
  const int wstride = L.max_cols * D;               // one system's columns of this CTA
  zc* const ub = (zc*)dsm;                          // [2][S][max_bond][D]
  zc* const w = ub + (size_t)2 * S * ustride;       // [S][max_cols][D]
  zc* const qb = w + (size_t)S * wstride;           // [2][S][2][D][D]
  zc* const ab = qb + (size_t)4 * S * DD;           // [2][stage]
  const int N = L.num_steps;
  auto columns = [&](int2 dm, int& c0, int& nc) {   // [c0, c0 + nc) of the r + 1 (the last one is B)
    const int per = (dm.y + C) / C;
    c0 = c * per;
    nc = max(0, min(per, dm.y + 1 - c0));
  };
  auto load_q = [&](int k) {
    const zc* src = (const zc*)L.qtab + ((long long)(L.pidx ? k : 0) * L.nh + h0) * 2 * DD;
    zc* dst = qb + (size_t)(k & 1) * 2 * S * DD;
    for (int idx = tid; idx < ns * 2 * DD; idx += nt) copy16(dst + idx, src + idx);
  };
  int2 dm = L.dims[0], dn = N > 1 ? L.dims[1] : dm;
  int c0, nc;
  columns(dm, c0, nc);
  if (L.stage) stage_columns(L, 0, dm, c0, nc, ab);
  load_q(0);
  // u_0 = P1_0 rho0, rho(0) = rho0 cap_0
  for (int idx = tid; idx < ns * D; idx += nt) {
    const int s = idx / D, a = idx - s * D, h = h0 + s;
    const zc* P1 = (const zc*)L.ptab + (long long)(L.pidx ? L.pidx[(long long)h * N] : h) * 2 * DD;
    const zc* r0 = (const zc*)L.rho0 + (long long)h * D;
    zc acc = mk<double>(0, 0);
    for (int b = 0; b < D; ++b) cfma(acc, P1[a * D + b], r0[b]);
    ub[(size_t)s * ustride + a] = acc;
    if (c == 0) {
      ((zc*)L.out)[(long long)h * D + a] = cmul(r0[a], ((const zc*)L.caps)[0]);
      if (RECORD) ((zc*)L.fwd_hist)[(long long)h * N * L.cap * D + a] = r0[a];
    }
  }
  copies_done();
  cluster.sync();   // also: every CTA of the cluster has started before its shared memory is written
  for (int k = 0; k < N; ++k) {
    const int l = dm.x, r = dm.y;
    const zc* u = ub + (size_t)(k & 1) * S * ustride;
    zc* un = ub + (size_t)((k + 1) & 1) * S * ustride;
    const zc* q = qb + (size_t)(L.pidx ? k & 1 : 0) * 2 * S * DD;
    const zc* as = ab + (size_t)(k & 1) * L.stage;
    int c0n = 0, ncn = 0;
    int2 dnn = dn;
    if (k + 1 < N) {
      columns(dn, c0n, ncn);
      if (L.stage) stage_columns(L, k + 1, dn, c0n, ncn, ab + (size_t)((k + 1) & 1) * L.stage);
      if (L.pidx) load_q(k + 1);
      if (k + 2 < N) dnn = L.dims[k + 2];
    }
    const int outs = nc * D;
    const int V = sum_parts(l, (r + 1) * D), G = WIDE ? part_lanes(V, outs) : V, parts = V / G;
    const int g = tid & (G - 1);
    for (int o0 = 0; o0 < outs; o0 += nt / G) {
      const int o = o0 + tid / G;
      const bool act = o < outs;
      const int cc = act ? o / D : 0, a = act ? o - cc * D : 0;
      zc sum[S];
#pragma unroll
      for (int s = 0; s < S; ++s) sum[s] = mk<double>(0, 0);
      if (act) {
        const bool last = c0 + cc == r;
        const zc* col = L.stage ? as + a * nc + cc
                        : last  ? (const zc*)L.bcol + (long long)k * L.cap * D + a
                                : (const zc*)L.sites + (long long)k * L.slot_elems + (size_t)a * r + c0 + cc;
        const size_t step = (size_t)D * (L.stage ? nc : last ? 1 : r);
        zc hold[WIDE ? S : 1];
#pragma unroll 1
        for (int j = 0; j < (WIDE ? parts : 1); ++j) {
          zc acc[S];
#pragma unroll
          for (int s = 0; s < S; ++s) acc[s] = mk<double>(0, 0);
          for (int l0 = WIDE ? part_index(j, g, G, parts) : g; l0 < l; l0 += 4 * V) {
            zc x[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
              if (l0 + t * V < l) x[t] = col[(l0 + t * V) * step];
#pragma unroll
            for (int t = 0; t < 4; ++t)
              if (l0 + t * V < l) {
#pragma unroll
                for (int s = 0; s < S; ++s) cfma(acc[s], u[(size_t)s * ustride + (l0 + t * V) * D + a], x[t]);
              }
          }
#pragma unroll
          for (int s = 0; s < S; ++s)
            if (WIDE)
              add_part(j, acc[s], sum[s], hold[s]);
            else
              sum[s] = acc[s];
        }
      }
#pragma unroll
      for (int s = 0; s < S; ++s) lane_sum(sum[s], G);
      if (act && g == 0)
#pragma unroll
        for (int s = 0; s < S; ++s) w[(size_t)s * wstride + cc * D + a] = sum[s];
    }
    __syncthreads();
    // the next states (to every CTA of the cluster) and the read-out
    for (int i = tid; i < (RECORD ? 2 : ns) * outs; i += nt) {
      const int s = RECORD || S > 1 ? i / outs : 0, o = i - s * outs;   // RECORD: s = 1 for v_{k+1}
      const int cc = o / D, a = o - cc * D;
      const bool last = c0 + cc == r, keep = RECORD && s == 1;
      if (keep && (last || k + 1 == N)) continue;
      const zc* M = q + (RECORD ? 0 : (size_t)s * 2 * DD) + a * D;
      const zc* x = w + (RECORD ? 0 : (size_t)s * wstride) + cc * D;
      const zc y = row_product(last || keep ? M + DD : M, 1, x, D);
      if (last) {
        ((zc*)L.out)[((long long)(k + 1) * L.nh + h0 + s) * D + a] = y;
        continue;
      }
      if (keep) {   // v_{k+1} = d P2_k w
        ((zc*)L.fwd_hist)[(((long long)h0 * N + k + 1) * L.cap + c0 + cc) * D + a] = y;
        continue;
      }
      zc* dst = un + (size_t)s * ustride + (size_t)(c0 + cc) * D + a;
      if (C == 1)
        *dst = y;
      else
        for (int t = 0; t < C; ++t) *cluster.map_shared_rank(dst, t) = y;
    }
    copies_done();
    if (C == 1)
      __syncthreads();
    else
      cluster.sync();
    dm = dn;
    dn = dnn;
    c0 = c0n;
    nc = ncn;
  }
}

// Adjoint sweep of compute_gradient_and_dynamics (gradient.py:323-425): from
// Y_{k+1} (bond r) to Y_k (bond l) through the transposed step,
//     w[l][b]   = sum_r A_k[l][b][r] z[r][b],   z[r][c] = d sum_e P2_k[e][c] Y_{k+1}[r][e]
//     Y_k[l][a] = sum_b P1_k[b][a] w[l][b]
// with the same propagator pairs as the forward sweep (controls and
// transforms folded in), so Y_k equals the reference's backward node before
// the pre-measurement control of step k.  As sweep_kernel, one system per
// cluster; the next z is (Q_{k-1})^T w.
template <int DT, bool WIDE>
__global__ void __launch_bounds__(SWEEP_THREADS, sweep_ctas(WIDE, DT)) sweep_back_kernel(SweepLaunch L, const double* target) {
  extern __shared__ __align__(16) unsigned char dsm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), c = (int)cluster.block_rank();
  const int D = DT ? DT : L.D, DD = D * D;
  const int tid = threadIdx.x;
  constexpr int nt = SWEEP_THREADS;
  const int h = (int)(blockIdx.x / C);
  const int zstride = L.max_bond * D;
  zc* const zb = (zc*)dsm;                           // [2][max_bond][D]
  zc* const w = zb + (size_t)2 * zstride;            // [max_cols][D]
  zc* const qb = w + (size_t)L.max_cols * D;         // [2][P1_k, Q_{k-1}][D][D]
  zc* const ab = qb + (size_t)4 * DD;                // [2][stage]
  const int N = L.num_steps;
  zc* const Y = (zc*)L.back_hist + (long long)h * (N + 1) * L.cap * D;
  auto q_of = [&](int k) { return (const zc*)L.qtab + ((long long)(L.pidx ? k : 0) * L.nh + h) * 2 * DD; };
  auto rows = [&](int2 dm, int& l0, int& nl) {       // this CTA's rows [l0, l0 + nl) of the l
    const int per = (dm.x + C - 1) / C;
    l0 = c * per;
    nl = max(0, min(per, dm.x - l0));
  };
  auto prefetch = [&](int k, int2 dm, int l0, int nl) {
    const zc* P1 = (const zc*)L.ptab + (long long)(L.pidx ? L.pidx[(long long)h * N + k] : h) * 2 * DD;
    const zc* Qp = q_of(k - 1);
    zc* qd = qb + (size_t)(k & 1) * 2 * DD;
    for (int idx = tid; idx < DD; idx += nt) {
      copy16(qd + idx, P1 + idx);
      copy16(qd + DD + idx, Qp + idx);
    }
    if (L.stage) {
      const zc* A = (const zc*)L.sites + (long long)k * L.slot_elems + (size_t)l0 * D * dm.y;
      zc* to = ab + (size_t)(k & 1) * L.stage;
      for (int e = tid; e < nl * D * dm.y; e += nt) copy16(to + e, A + e);
    }
  };
  int2 dm = L.dims[N - 1], dn = N > 1 ? L.dims[N - 2] : dm;
  int l0, nl;
  rows(dm, l0, nl);
  if (N > 1) prefetch(N - 1, dm, l0, nl);
  // z_{N-1} = d P2_{N-1}^T target (bond 1)
  for (int a = tid; a < D; a += nt) {
    const zc* t = (const zc*)target + (long long)h * D;
    const zc* P2d = q_of(N - 1) + DD;
    zc acc = mk<double>(0, 0);
    for (int e = 0; e < D; ++e) cfma(acc, P2d[e * D + a], t[e]);
    zb[(size_t)((N - 1) & 1) * zstride + a] = acc;
    if (c == 0) Y[(long long)N * L.cap * D + a] = t[a];
  }
  copies_done();
  cluster.sync();
  for (int k = N - 1; k >= 1; --k) {
    const int r = dm.y;
    const zc* z = zb + (size_t)(k & 1) * zstride;
    zc* zn = zb + (size_t)((k - 1) & 1) * zstride;
    const zc* q = qb + (size_t)(k & 1) * 2 * DD;
    int l0n = 0, nln = 0;
    int2 dnn = dn;
    if (k > 1) {
      rows(dn, l0n, nln);
      prefetch(k - 1, dn, l0n, nln);
      if (k > 2) dnn = L.dims[k - 2];
    }
    const zc* base = L.stage ? ab + (size_t)(k & 1) * L.stage
                             : (const zc*)L.sites + (long long)k * L.slot_elems + (size_t)l0 * D * r;
    const int outs = nl * D;
    const int V = sum_parts(r, dm.x * D), G = WIDE ? part_lanes(V, outs) : V, parts = V / G;
    const int g = tid & (G - 1);
    for (int o0 = 0; o0 < outs; o0 += nt / G) {
      const int o = o0 + tid / G;
      const bool act = o < outs;
      zc sum = mk<double>(0, 0);
      if (act) {
        const int b = o % D;
        const zc* row = base + (size_t)o * r;
        zc hold;
#pragma unroll 1
        for (int j = 0; j < (WIDE ? parts : 1); ++j) {
          zc acc = mk<double>(0, 0);
          for (int r0 = WIDE ? part_index(j, g, G, parts) : g; r0 < r; r0 += 4 * V) {
            zc x[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
              if (r0 + t * V < r) x[t] = row[r0 + t * V];
#pragma unroll
            for (int t = 0; t < 4; ++t)
              if (r0 + t * V < r) cfma(acc, x[t], z[(r0 + t * V) * D + b]);
          }
          if (WIDE)
            add_part(j, acc, sum, hold);
          else
            sum = acc;
        }
      }
      lane_sum(sum, G);
      if (act && g == 0) w[o] = sum;
    }
    __syncthreads();
    for (int o = tid; o < 2 * outs; o += nt) {
      const bool next = o >= outs;
      const int i = next ? o - outs : o;
      const int li = i / D, a = i - li * D;
      const zc acc = row_product(q + (next ? DD : 0) + a, D, w + li * D, D);
      if (!next) {
        Y[((long long)k * L.cap + l0 + li) * D + a] = acc;
        continue;
      }
      zc* dst = zn + (size_t)(l0 + li) * D + a;
      if (C == 1)
        *dst = acc;
      else
        for (int t = 0; t < C; ++t) *cluster.map_shared_rank(dst, t) = acc;
    }
    copies_done();
    if (C == 1)
      __syncthreads();
    else
      cluster.sync();
    dm = dn;
    dn = dnn;
    l0 = l0n;
    nl = nln;
  }
}

// Derivative cores: for every step n and system h,
//     core[n][a][m][e] = sum_{l, r} v_n[l][a] T_n[l][r][m] Y_{n+1}[r][e]
// (T_n = d * site_n, diagonal in its system legs), first
// X[r][a][m] = sum_l v_n[l][a] T_n[l][r][m] in shared memory, then the sum
// over r.  The host maps a core to the reference's derivative tensor (the
// post-measurement control of step n on leg a, the pre-measurement control
// of step n+1 on leg e, the process tensor's transforms on the MPO legs).
// Grid: (steps, systems).
__global__ void __launch_bounds__(DYN_THREADS) dyn_deriv_kernel(SweepLaunch L) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const int n = blockIdx.x;
  const int h = blockIdx.y;
  const int D = L.D;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int2 dm = L.dims[n];
  const int l = dm.x, r = dm.y;
  const zc* A = (const zc*)L.sites + (long long)n * L.slot_elems;
  const zc* v = (const zc*)L.fwd_hist + ((long long)h * L.num_steps + n) * L.cap * D;
  const zc* Y = (const zc*)L.back_hist + ((long long)h * (L.num_steps + 1) + n + 1) * L.cap * D;
  zc* X = (zc*)dsm;   // r * D * D
  for (int idx = tid; idx < r * D * D; idx += nt) {
    const int rr = idx / (D * D), am = idx - rr * D * D;
    const int a = am / D, m = am - a * D;
    zc acc = mk<double>(0, 0);
    for (int ll = 0; ll < l; ++ll) cfma(acc, v[ll * D + a], A[((size_t)ll * D + m) * r + rr]);
    X[idx] = cscale(acc, (double)L.d);
  }
  __syncthreads();
  zc* out = (zc*)L.deriv + ((long long)h * L.num_steps + n) * D * D * D;
  for (int idx = tid; idx < D * D * D; idx += nt) {
    const int a = idx / (D * D), me = idx - a * D * D;
    const int m = me / D, e = me - m * D;
    zc acc = mk<double>(0, 0);
    for (int rr = 0; rr < r; ++rr) cfma(acc, X[((size_t)rr * D + a) * D + m], Y[rr * D + e]);
    out[idx] = acc;
  }
}

// Shape of a sweep: systems per CTA, CTAs per cluster, dynamic shared memory.
// Many systems: one CTA per SM with its share of them (every load of A serves
// all of a CTA's systems).  Few: the step's columns are split over up to eight
// CTAs while a CTA's FP64 work of a step (2 l r D clocks on one SM) is above
// 3000 clocks (bond 20 with D = 4).  8 systems, 60 steps, whole calls on 1 / 2 /
// 4 / 8 CTAs each, sweep and gradient in us: bond 9 202 224 213 215, 390 436 436
// 437; bond 15 252 249 240 236, 474 474 472 475; bond 37 673 487 398 393, 1381 969
// 783 769; bond 112 2955 1661 948 611, 6834 4102 2715 1995.  Below the line the
// cluster's barrier takes what the split saves.
// Two CTAs each as well from half a system to one and a half per SM, where the
// columns of half a step are too wide to stage (bond 54 on with D = 4, 37 with
// D = 9), so that several CTAs fit on an SM: a whole system more on one SM than
// on the next doubles the call, half a one adds a half.  60 steps, bond 60 and 90,
// one CTA (above 152 systems two systems each) -> two: 77 systems 962 1956 -> 959
// 1663, 152 systems 1002 1979 -> 984 1692, 153 systems 1701 3412 -> 1355 2406, 228
// systems 1710 3421 -> 1369 2425; 230 systems 1714 3421 -> 1797 3266.  Gradients,
// bond 90: 77 systems 7095 -> 6503, 153 systems 11990 -> 10720.  D = 9, bond 55: 77
// systems 789 -> 778, 153 systems 1431 -> 1195.  Staged columns (bond 36): 153
// systems 990 -> 1014, 190 systems 996 -> 1269.
struct SweepShape {
  int S, C, max_cols;
  size_t stage;   // elements of one staging buffer, 0 = columns read from global memory
  size_t smem;
};

static SweepShape sweep_shape(const SweepLaunch& L, int max_s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  sms = sms > 0 ? sms : 1;
  const size_t limit = 200 * 1024;
  const auto cols = [&](int C) { return (L.max_bond + C) / C; };
  const auto bytes = [&](int S, int C) {
    return ((size_t)2 * S * L.max_bond * L.D + (size_t)S * cols(C) * L.D + (size_t)4 * S * L.D * L.D) * sizeof(zc);
  };
  const auto stage = [&](int C) { return (size_t)L.max_bond * L.D * cols(C); };
  const auto staged = [&](int S, int C) { return bytes(S, C) + 2 * stage(C) * sizeof(zc) <= limit; };
  SweepShape sh;
  const double clocks = 2.0 * L.max_bond * L.max_bond * L.D;
  sh.C = 1;
  while (sh.C < 8 && 2 * sh.C * L.nh <= sms && clocks > 3000.0 * sh.C) sh.C *= 2;
  if (2 * L.nh > sms && 2 * L.nh <= 3 * sms && clocks > 3000.0 && !staged(1, 2)) sh.C = 2;
  sh.S = sh.C > 1 ? 1 : std::min(max_s, (L.nh + sms - 1) / sms);
  while (sh.S > 1 && bytes(sh.S, sh.C) > limit) --sh.S;
  sh.max_cols = cols(sh.C);
  sh.smem = bytes(sh.S, sh.C);
  sh.stage = staged(sh.S, sh.C) ? stage(sh.C) : 0;
  sh.smem += 2 * sh.stage * sizeof(zc);
  return sh;
}

template <typename K, typename... Args>
static cudaError_t launch_clusters(K kernel, int ctas, int C, size_t smem, cudaStream_t stream, Args... args) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(SWEEP_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t launch_sweep_prepare(const SweepLaunch& L, cudaStream_t stream) {
  // enough CTAs per step for its columns; step 0's also form the propagators
  const int y = std::max(1, std::min(64, std::max((L.cap * L.D * 8) / SWEEP_THREADS / 4,
                                                  (L.nh * L.D * L.D + SWEEP_THREADS - 1) / SWEEP_THREADS / 2)));
  sweep_prepare_kernel<<<dim3(L.num_steps, y), SWEEP_THREADS, 0, stream>>>(L);
  return cudaGetLastError();
}

// Has any step more columns than lanes for its partial sums (WIDE)?
bool sweep_is_wide(int D, int num_steps, const int2* dims) {
  for (int k = 0; k < num_steps; ++k) {
    const int fwd = (dims[k].y + 1) * D, back = dims[k].x * D;
    const int vf = sum_parts(dims[k].x, fwd), vb = sum_parts(dims[k].y, back);
    if (part_lanes(vf, fwd) < vf || part_lanes(vb, back) < vb) return true;
  }
  return false;
}

template <int DT, bool WIDE>
static cudaError_t launch_sweep_shape(const SweepLaunch& L, const SweepShape& sh, cudaStream_t stream) {
  const int ctas = (L.nh + sh.S - 1) / sh.S * sh.C;
  if (L.fwd_hist) return launch_clusters(sweep_kernel<1, true, DT, WIDE>, ctas, sh.C, sh.smem, stream, L);
  switch (sh.S) {
    case 1: return launch_clusters(sweep_kernel<1, false, DT, WIDE>, ctas, sh.C, sh.smem, stream, L);
    case 2: return launch_clusters(sweep_kernel<2, false, DT, WIDE>, ctas, sh.C, sh.smem, stream, L);
    case 4: return launch_clusters(sweep_kernel<4, false, DT, WIDE>, ctas, sh.C, sh.smem, stream, L);
  }
  if constexpr (DT == 4) {
    switch (sh.S) {
      case 3: return launch_clusters(sweep_kernel<3, false, 4, WIDE>, ctas, sh.C, sh.smem, stream, L);
      case 5: return launch_clusters(sweep_kernel<5, false, 4, WIDE>, ctas, sh.C, sh.smem, stream, L);
      case 6: return launch_clusters(sweep_kernel<6, false, 4, WIDE>, ctas, sh.C, sh.smem, stream, L);
      case 7: return launch_clusters(sweep_kernel<7, false, 4, WIDE>, ctas, sh.C, sh.smem, stream, L);
      case 8: return launch_clusters(sweep_kernel<8, false, 4, WIDE>, ctas, sh.C, sh.smem, stream, L);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_sweep(const SweepLaunch& L0, cudaStream_t stream) {
  SweepLaunch L = L0;
  SweepShape sh = sweep_shape(L, L.fwd_hist ? 1 : L.D == 4 ? 8 : 4);
  if (L.D != 4 && sh.S == 3) sh = sweep_shape(L, 2);   // built for 1, 2 and 4 systems
  L.max_cols = sh.max_cols;
  L.stage = (long long)sh.stage;
  if (L.D == 4) return L.wide ? launch_sweep_shape<4, true>(L, sh, stream) : launch_sweep_shape<4, false>(L, sh, stream);
  return L.wide ? launch_sweep_shape<0, true>(L, sh, stream) : launch_sweep_shape<0, false>(L, sh, stream);
}

cudaError_t launch_sweep_back(const SweepLaunch& L0, const double* target, cudaStream_t stream) {
  SweepLaunch L = L0;
  const SweepShape sh = sweep_shape(L, 1);
  L.max_cols = sh.max_cols;
  L.stage = (long long)sh.stage;
  const int ctas = L.nh * sh.C;
  if (L.D == 4)
    return L.wide ? launch_clusters(sweep_back_kernel<4, true>, ctas, sh.C, sh.smem, stream, L, target)
                  : launch_clusters(sweep_back_kernel<4, false>, ctas, sh.C, sh.smem, stream, L, target);
  return L.wide ? launch_clusters(sweep_back_kernel<0, true>, ctas, sh.C, sh.smem, stream, L, target)
                : launch_clusters(sweep_back_kernel<0, false>, ctas, sh.C, sh.smem, stream, L, target);
}

cudaError_t launch_dyn_deriv(const SweepLaunch& L, cudaStream_t stream) {
  const size_t smem = (size_t)L.max_bond * L.D * L.D * sizeof(zc);
  cudaError_t e = cudaFuncSetAttribute(dyn_deriv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid(L.num_steps, L.nh);
  dyn_deriv_kernel<<<grid, DYN_THREADS, smem, stream>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_dyn_step(const DynLaunch& L, int r, cudaStream_t stream) {
  const int chunks = (r + DYN_RB - 1) / DYN_RB;
  const size_t smem = (size_t)(L.cap * L.D + 2 * DYN_RB * L.D) * sizeof(zc);
  dim3 grid(chunks, L.nh);
  dyn_step_kernel<<<grid, DYN_THREADS, smem, stream>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_dyn_init(const DynLaunch& L, const double* rho0, cudaStream_t stream) {
  dyn_init_kernel<<<L.nh, 32, 0, stream>>>(L, rho0);
  return cudaGetLastError();
}

}  // namespace otb
