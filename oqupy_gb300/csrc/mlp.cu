// BF16 tensor-core GEMM (tcgen05, sm_103a) and the elementwise kernels of
// the MLP surrogate (forward, backward, AdamW).
//
//   C[M][N] = A[M][K] * B[N][K]^T      A, B bf16, K contiguous ("K-major")
//
// Operands with 16-byte aligned rows go through tc_gemm_tma_kernel (below),
// others through tc_gemm_pipe_kernel: one CTA (128 threads) computes a 128 x
// 128 tile.  Per 64-wide K chunk the CTA stages A and B into shared memory in the canonical no-swizzle K-major
// layout of the 5th-generation tensor core -- 8-row x 16-byte core matrices,
// the two core matrices of a 16-deep K step 128 B apart (leading byte
// offset), successive 8-row groups 1024 B apart (stride byte offset) -- and
// one elected thread issues four tcgen05.mma (M=128, N=128, K=16, bf16 in,
// FP32 accumulate) into a 128-column TMEM accumulator, then tcgen05.commit to
// an mbarrier.  Every wait on that mbarrier is bounded; on timeout the kernel
// records an error, still frees its TMEM and returns.  The epilogue reads the
// accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 = tile
// rows) and applies the fused bias / GELU / GELU-gradient step.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/oqupy_gb300.h"
#include "capi_util.h"

namespace otb {

constexpr int TC_BM = 128, TC_BN = 128, TC_BK = 64;
constexpr int TC_THREADS = 128;
constexpr long long TC_WAIT_LIMIT = 1LL << 26;

enum : int {
  EPI_NONE = 0,       // out = acc (+ bias)
  EPI_GELU = 1,       // z = acc + bias -> z_out (FP32), out = gelu(z)
  EPI_GELU_GRAD = 2,  // out = acc * gelu'(z_in)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor, no swizzle, K-major
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of the 5th-generation tensor core
  return d;                // base offset 0, layout: no swizzle
}

// instruction descriptor: kind::f16, A/B bf16, D f32, both K-major
__host__ __device__ constexpr uint32_t make_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// Stages a 128 x 64 bf16 tile (rows r0.., k k0..) of a row-major [R][K] matrix
// into the core-matrix layout, core (rg, kg) at (rg * 8 + kg) * 128 B: 16-byte
// cp.async copies (no register round trip) for every aligned full chunk;
// ragged or unaligned chunks (K % 8 != 0, tile edges) are zero-padded through
// registers.
__device__ __forceinline__ void stage_tile_async(unsigned char* dst, const __nv_bfloat16* src, int R, int K,
                                                 int r0, int k0) {
  for (int chunk = threadIdx.x; chunk < TC_BM * (TC_BK / 8); chunk += blockDim.x) {
    const int rr = chunk / (TC_BK / 8), kc = chunk % (TC_BK / 8);
    const int row = r0 + rr, kk = k0 + kc * 8;
    const int rg = rr >> 3, r8 = rr & 7;
    unsigned char* d = dst + (size_t)(rg * (TC_BK / 8) + kc) * 128 + r8 * 16;
    const __nv_bfloat16* p = src + (size_t)row * K + kk;
    if (row < R && kk + 8 <= K && ((reinterpret_cast<uintptr_t>(p) & 15) == 0)) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(d)), "l"(p) : "memory");
    } else {
      union {
        uint4 u;
        __nv_bfloat16 h[8];
      } tmp;
      tmp.u = make_uint4(0, 0, 0, 0);
      if (row < R)
        for (int e = 0; e < 8; ++e)
          if (kk + e < K) tmp.h[e] = p[e];
      *reinterpret_cast<uint4*>(d) = tmp.u;
    }
  }
}

struct GemmOut {
  const float* bias;
  const float* zin;
  float* zout;
  float* outf;
  __nv_bfloat16* outb;
  int ldf;   // row stride of zin, zout and outf
  int ldb;   // row stride of outb
  int epi;
};

// n <= 16 consecutive outputs of one row, in the widest stores the address allows.
__device__ __forceinline__ void store16(float* p, const float* v, int n) {
  if (n == 16 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      reinterpret_cast<float4*>(p)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q < n) p[q] = v[q];
  }
}
__device__ __forceinline__ void store16(__nv_bfloat16* p, const float* v, int n) {
  if (n == 16 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    union {
      uint4 u[2];
      __nv_bfloat162 h[8];
    } t;
#pragma unroll
    for (int q = 0; q < 8; ++q) t.h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
    reinterpret_cast<uint4*>(p)[0] = t.u[0];
    reinterpret_cast<uint4*>(p)[1] = t.u[1];
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q < n) p[q] = __float2bfloat16(v[q]);
  }
}

// The fused step on CH accumulators of one row (n of them inside the matrix):
// v = the outputs; with EPI_GELU z = the pre-activations.
template <int CH>
__device__ __forceinline__ void fused_step(const GemmOut& o, const uint32_t* r, size_t at, int col, int n, float* v,
                                           float* z) {
#pragma unroll
  for (int q = 0; q < CH; ++q) v[q] = __uint_as_float(r[q]);
  if (o.epi == EPI_GELU_GRAD) {
    const float* zi = o.zin + at;
    if (n == CH && (reinterpret_cast<uintptr_t>(zi) & 15) == 0) {
#pragma unroll
      for (int q = 0; q < CH / 4; ++q) {
        const float4 t = reinterpret_cast<const float4*>(zi)[q];
        v[4 * q] *= gelu_grad_f(t.x);
        v[4 * q + 1] *= gelu_grad_f(t.y);
        v[4 * q + 2] *= gelu_grad_f(t.z);
        v[4 * q + 3] *= gelu_grad_f(t.w);
      }
    } else {
#pragma unroll
      for (int q = 0; q < CH; ++q)
        if (q < n) v[q] *= gelu_grad_f(zi[q]);
    }
    return;
  }
  if (o.bias) {
#pragma unroll
    for (int q = 0; q < CH; ++q)
      if (q < n) v[q] += __ldg(o.bias + col + q);
  }
  if (o.epi == EPI_GELU) {
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      z[q] = v[q];
      v[q] = gelu_f(v[q]);
    }
  }
}

// 16 accumulators of one row through the fused step and to memory.
__device__ __forceinline__ void epilogue16(const GemmOut& o, const uint32_t* r, size_t row, int col, int n) {
  float v[16], z[16];
  const size_t at = row * o.ldf + col;
  fused_step<16>(o, r, at, col, n, v, z);
  if (o.epi == EPI_GELU && o.zout) store16(o.zout + at, z, n);
  if (o.outf) store16(o.outf + at, v, n);
  if (o.outb) store16(o.outb + row * o.ldb + col, v, n);
}

__device__ __forceinline__ bool tc_wait_phase(uint64_t* mbar, int phase) {
  uint32_t done = 0;
  for (long long it = 0; it < TC_WAIT_LIMIT && !done; ++it) {
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(mbar)), "r"(phase));
  }
  return done != 0;
}

// Two-stage pipeline: while the tensor core runs the four MMAs of chunk k, the CTA's cp.async copies of chunk k+1 land in
// the other buffer.  A buffer is refilled only after the mbarrier reports
// the MMAs that read it complete (at most one MMA batch is outstanding at
// any wait, so the phase parity identifies it).  All waits are bounded.
__global__ void __launch_bounds__(TC_THREADS)
    tc_gemm_pipe_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, int M, int N,
                        int K, const float* __restrict__ bias, int epi, const float* __restrict__ zin,
                        float* __restrict__ zout, float* __restrict__ outf, __nv_bfloat16* __restrict__ outb,
                        int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char tc_dsm[];
  unsigned char* sA[2] = {tc_dsm, tc_dsm + TC_BM * TC_BK * 2};
  unsigned char* sB[2] = {tc_dsm + 2 * TC_BM * TC_BK * 2, tc_dsm + 2 * TC_BM * TC_BK * 2 + TC_BN * TC_BK * 2};
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  __shared__ int s_err;
  __shared__ int s_drain;  // phase parity of an MMA batch still in flight after a timed-out wait
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * TC_BN;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(TC_BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)));
    asm volatile("fence.mbarrier_init.release.cluster;");
    s_err = 0;
    s_drain = -1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = make_idesc(TC_BM, TC_BN);

  const int nk = (K + TC_BK - 1) / TC_BK;
  stage_tile_async(sA[0], A, M, K, m0, 0);
  stage_tile_async(sB[0], B, N, K, n0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  int issued = 0;   // MMA batches committed so far (batch j completes phase j & 1)
  for (int kc = 0; kc < nk; ++kc) {
    const int buf = kc & 1;
    if (kc >= 1) {
      // batch kc - 1 read the other buffer: wait for it before refilling, and
      // so that no more than one batch is outstanding at any parity wait
      if (tid == 0 && !s_err && !tc_wait_phase(&mbar, (kc - 1) & 1)) {
        s_err = 1;
        s_drain = (kc - 1) & 1;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      __syncthreads();
      if (s_err) break;
    }
    if (kc + 1 < nk) {
      stage_tile_async(sA[buf ^ 1], A, M, K, m0, (kc + 1) * TC_BK);
      stage_tile_async(sB[buf ^ 1], B, N, K, n0, (kc + 1) * TC_BK);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      for (int ks = 0; ks < TC_BK / 16; ++ks) {
        const uint64_t ad = make_desc(smem_u32(sA[buf]) + ks * 2 * 128, 128, (TC_BK / 8) * 128);
        const uint64_t bd = make_desc(smem_u32(sB[buf]) + ks * 2 * 128, 128, (TC_BK / 8) * 128);
        const uint32_t acc = (kc > 0 || ks > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(&mbar)));
    }
    ++issued;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // the last committed batch: every earlier one was waited for in the loop
  if (tid == 0 && !s_err && issued > 0 && !tc_wait_phase(&mbar, (issued - 1) & 1)) {
    s_err = 1;
    s_drain = (issued - 1) & 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");

  if (!s_err) {
    const GemmOut o{bias, zin, zout, outf, outb, N, N, epi};
    const int row = m0 + warp * 32 + lane;
    for (int c0 = 0; c0 < TC_BN; c0 += 16) {
      uint32_t r[16];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + c0;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;");
      if (row < M && n0 + c0 < N) epilogue16(o, r, (size_t)row, n0 + c0, min(16, N - n0 - c0));
    }
  } else if (tid == 0) {
    atomicExch(err, 1);
    // one more bounded wait for the batch still in flight, so that it is
    // not writing the accumulator when the columns are released
    if (s_drain >= 0) tc_wait_phase(&mbar, s_drain);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_BN));
  }
}

// ---------------------------------------------------------------------------
// TMA-fed persistent GEMM
// ---------------------------------------------------------------------------
//
// Every CTA (one per SM) walks over 128 x BN tiles: one warp issues the TMA
// loads of 64-deep K chunks into a ring of shared-memory stages (128-byte
// swizzle), one thread issues the tcgen05.mma, eight warps run the epilogue
// from TMEM, where two accumulators let the next tile's products overlap it.
// Either operand may be stored K-contiguous ([rows][K]) or transposed
// ([K][rows], the tensor core's MN-major layout), so that weight gradients read
// activations and their gradients as they lie.
//
// What bounds it: for the hidden layers the epilogue's FP32 issue (GELU: about
// 45 instructions an output, eight warps), for a wide output layer the FP32
// result's write to memory.  The two-stage kernel above (cp.async staging by
// the warps that also issue the products and run the epilogue, scalar stores)
// reached 79 TFLOP/s on a 60001-point inference of a 5-512x4-1500 network
// (2370 us); with this one the inference takes 438 us.  bf16 rows and
// pre-activations are stored by the lane that holds them (a 512-wide hidden
// layer takes 72 us, 78 through shared memory), FP32 results through shared
// memory as whole row segments (output layer 144 us, 190 without).  A training
// step of 256 points, where the 1500-column operands were staged element by
// element and both operands of every weight gradient transposed first: 1020 ->
// 330 us, launches 45 -> 19.
//
// Used when rows are 16-byte aligned; other operands keep the kernel above.
// Tile width: 256 where that gives every SM a tile, else 128, else 64 (a
// training step's products have few tiles, and are bound by one tile's chain).
constexpr int TM_BM = 128, TM_BK = 64;
constexpr int TM_EPI_WARPS = 8;
constexpr int TM_THREADS = 64 + 32 * TM_EPI_WARPS;
constexpr unsigned long long TM_WAIT_NS = 2000000000ull;

constexpr int TM_XPOSE = 32 * 33 * 4;   // an epilogue warp's transposition buffer (rows 33 words apart)

template <int BN>
struct TmShape {
  static constexpr int stages = BN == 256 ? 3 : 5;
  static constexpr int a_bytes = TM_BM * TM_BK * 2;
  static constexpr int b_bytes = BN * TM_BK * 2;
  static constexpr int ring = stages * (a_bytes + b_bytes);
  static constexpr int smem = ring + TM_EPI_WARPS * TM_XPOSE + 1024;   // + alignment
  static constexpr int tmem_cols = 2 * BN;
};

// shared-memory matrix descriptor, 128-byte swizzle; K-major: 8-row groups
// 1024 B apart; MN-major: 64-wide column blocks 8192 B apart (64 K rows of 128
// B each), 8-row K groups 1024 B apart
__device__ __forceinline__ uint64_t swizzled_desc(uint32_t saddr, bool mn_major) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((mn_major ? 8192 : 16) >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__device__ __forceinline__ void tma_load(const CUtensorMap* map, uint64_t* bar, uint32_t dst, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// Wait bounded to TM_WAIT_NS, which also ends when another role has given up.
__device__ __forceinline__ bool tm_wait(uint64_t* bar, int parity, volatile int* abort) {
  unsigned long long t0 = 0, t;
  for (int it = 0;; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if (*abort) return false;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (it == 0) t0 = t;
    if (t - t0 > TM_WAIT_NS) break;
  }
  *abort = 1;
  return false;
}

// Waits (bounded) for the last use of every stage after `used` uses in turn.
__device__ __forceinline__ void tm_drain(uint64_t* bars, int stages, int used) {
  for (int st = 0; st < stages && st < used; ++st) {
    int never = 0;
    tm_wait(&bars[st], ((used - st + stages - 1) / stages - 1) & 1, &never);
  }
}

__device__ __forceinline__ void tm_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int BN>
__global__ void __launch_bounds__(TM_THREADS, 1)
    tc_gemm_tma_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int M, int N,
                       int K, int ta, int tb, GemmOut out, int* __restrict__ err) {
  typedef TmShape<BN> Sh;
  extern __shared__ unsigned char tm_raw[];
  __shared__ __align__(8) uint64_t full[Sh::stages], empty[Sh::stages], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const uint32_t base = (smem_u32(tm_raw) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(Sh::tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < Sh::stages; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[i])));
    }
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&acc_full[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acc_empty[i])), "r"(TM_EPI_WARPS));
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
    abort_flag = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  volatile int* const stop = &abort_flag;
  const int nk = (K + TM_BK - 1) / TM_BK;
  const int tn = (N + BN - 1) / BN, tiles = tn * ((M + TM_BM - 1) / TM_BM);
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // this CTA's tiles

  if (warp == 0 && lane == 0) {
    int it = 0;   // chunk counter: stage it % stages, use it / stages
    for (int t = 0; t < mine && !*stop; ++t) {
      const int tile = blockIdx.x + t * gridDim.x;
      const int m0 = tile / tn * TM_BM, n0 = tile % tn * BN;
      for (int kc = 0; kc < nk; ++kc, ++it) {
        const int st = it % Sh::stages, use = it / Sh::stages;
        if (use > 0 && !tm_wait(&empty[st], (use - 1) & 1, stop)) break;
        const uint32_t sa = base + st * (Sh::a_bytes + Sh::b_bytes), sb = sa + Sh::a_bytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[st])),
                     "r"(Sh::a_bytes + Sh::b_bytes)
                     : "memory");
        if (ta) {
          for (int j = 0; j < TM_BM / 64; ++j) tma_load(&mapA, &full[st], sa + j * 8192, m0 + 64 * j, kc * TM_BK);
        } else {
          tma_load(&mapA, &full[st], sa, kc * TM_BK, m0);
        }
        if (tb) {
          for (int j = 0; j < BN / 64; ++j) tma_load(&mapB, &full[st], sb + j * 8192, n0 + 64 * j, kc * TM_BK);
        } else {
          tma_load(&mapB, &full[st], sb, kc * TM_BK, n0);
        }
      }
    }
    // after a give-up: no copy may be in flight when the CTA ends
    if (*stop) tm_drain(full, Sh::stages, it);
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = make_idesc(TM_BM, BN) | (ta ? 1u << 15 : 0u) | (tb ? 1u << 16 : 0u);
    const int step_a = ta ? 2048 : 32, step_b = tb ? 2048 : 32;   // bytes of a 16-deep K step
    int it = 0;
    for (int t = 0; t < mine && !*stop; ++t) {
      const int buf = t & 1;
      if (t >= 2 && !tm_wait(&acc_empty[buf], ((t >> 1) - 1) & 1, stop)) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      bool ok = true;
      for (int kc = 0; kc < nk; ++kc, ++it) {
        const int st = it % Sh::stages;
        if (!tm_wait(&full[st], (it / Sh::stages) & 1, stop)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t sa = base + st * (Sh::a_bytes + Sh::b_bytes), sb = sa + Sh::a_bytes;
#pragma unroll
        for (int ks = 0; ks < TM_BK / 16; ++ks) {
          const uint64_t ad = swizzled_desc(sa + ks * step_a, ta), bd = swizzled_desc(sb + ks * step_b, tb);
          const uint32_t acc = (kc > 0 || ks > 0) ? 1u : 0u;
          asm volatile(
              "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
              " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem + buf * BN),
              "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(&empty[st])));
      }
      if (!ok) break;
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(&acc_full[buf])));
    }
    // after a give-up: no product may be in flight when TMEM is released
    if (*stop) tm_drain(empty, Sh::stages, it);
  } else if (warp >= 2) {
    const int quarter = warp & 3, half = (warp - 2) >> 2;   // TMEM lanes 32 quarter.., columns half
    for (int t = 0; t < mine; ++t) {
      const int buf = t & 1;
      const int tile = blockIdx.x + t * gridDim.x;
      const int m0 = tile / tn * TM_BM, n0 = tile % tn * BN;
      if (!__all_sync(0xffffffffu, tm_wait(&acc_full[buf], (t >> 1) & 1, stop))) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int row0 = m0 + quarter * 32, row = row0 + lane;
      const int rows = min(32, M - row0);
      float* const xbuf = reinterpret_cast<float*>(tm_raw + (base - smem_u32(tm_raw)) + Sh::ring) + (warp - 2) * (TM_XPOSE / 4);
      for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
        if (n0 + c0 >= N) break;
        uint32_t r[32];
        const uint32_t taddr = tmem + buf * BN + ((uint32_t)(quarter * 32) << 16) + c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;");
        if (rows <= 0) continue;
        const int col = n0 + c0;
        if (col + 32 <= N) {
          // bf16 rows and pre-activations as 32- and 64-byte pieces of the lane's
          // own row; FP32 results, twice the bytes, as whole row segments
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            float v[16], z[16];
            // rows past the matrix read row 0's pre-activations and are not stored
            fused_step<16>(out, r + 16 * hf, (size_t)(row < M ? row : row0) * out.ldf + col + 16 * hf, col + 16 * hf, 16, v, z);
            if (row < M) {
              if (out.epi == EPI_GELU && out.zout) store16(out.zout + (size_t)row * out.ldf + col + 16 * hf, z, 16);
              if (out.outb) store16(out.outb + (size_t)row * out.ldb + col + 16 * hf, v, 16);
            }
            if (out.outf) {
#pragma unroll
              for (int q = 0; q < 16; ++q) xbuf[lane * 33 + 16 * hf + q] = v[q];
            }
          }
          if (out.outf) {
            __syncwarp();
            float* dst = out.outf + (size_t)row0 * out.ldf + col + lane;
            for (int i = 0; i < rows; ++i) dst[(size_t)i * out.ldf] = xbuf[i * 33 + lane];
          }
        } else if (row < M) {
          epilogue16(out, r, (size_t)row, col, min(16, N - col));
          if (col + 16 < N) epilogue16(out, r + 16, (size_t)row, col + 16, N - col - 16);
        }
        __syncwarp();
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      if (lane == 0) tm_arrive(&acc_empty[buf]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (tid == 0 && abort_flag) atomicExch(err, 1);
  __syncwarp();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Sh::tmem_cols));
  }
}

// out[c][r] = in[r][c] (bf16), 32 x 32 tiles through shared memory
__global__ void transpose_bf16_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out,
                                      int R, int C) {
  __shared__ __nv_bfloat16 t[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    t[i][threadIdx.x] = (r < R && c < C) ? in[(size_t)r * C + c] : __float2bfloat16(0.f);
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (c < C && r < R) out[(size_t)c * R + r] = t[threadIdx.x][i];
  }
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(in[i]);
}

// column sums of a row-major [R][C] FP32 matrix (bias gradients)
__global__ void colsum_kernel(const float* __restrict__ in, float* __restrict__ out, int R, int C) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float s = 0.f;
  for (int r = 0; r < R; ++r) s += in[(size_t)r * C + c];
  out[c] = s;
}

// Bias gradients of every layer in one launch: column sums of row-major FP32
// matrices.  A CTA takes 32 columns of one matrix: 8 warps sum every eighth row
// (coalesced), then the eight partial sums in order.  (One thread per column on
// a handful of CTAs, one launch a layer: 17 us each for 256 rows; all of them
// now: 5 us.)
constexpr int MLP_MAX_LAYERS = 32;
struct ColsumJobs {
  int n, rows;
  int first[MLP_MAX_LAYERS + 1];   // first CTA of every matrix
  int cols[MLP_MAX_LAYERS];
  const float* in[MLP_MAX_LAYERS];
  float* out[MLP_MAX_LAYERS];
};

__global__ void __launch_bounds__(256) colsum_multi_kernel(const __grid_constant__ ColsumJobs j) {
  __shared__ float part[8][33];
  int q = 0;
  while (q + 1 < j.n && (int)blockIdx.x >= j.first[q + 1]) ++q;
  const int C = j.cols[q];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = ((int)blockIdx.x - j.first[q]) * 32 + lane;
  float s = 0.f;
  if (c < C) {
    const float* p = j.in[q] + c;
#pragma unroll 4
    for (int r = warp; r < j.rows; r += 8) s += p[(size_t)r * C];
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < C) {
#pragma unroll
    for (int w = 1; w < 8; ++w) s += part[w][lane];
    j.out[q][c] = s;
  }
}

// AdamW on every tensor of a network in one launch, 32 x 32 tiles; weights also
// refresh their bf16 copy (row stride ldw) and its transpose (row stride ldt).
// (Two updates and a transposition per layer, 15 launches of 3 to 8 us for five
// layers, before.)
struct AdamTensor {
  float *w, *m, *v;
  const float* g;
  __nv_bfloat16 *wb, *wt;   // null: a bias
  int rows, cols, ldw, ldt, first;
  float wd;
};
struct AdamJobs {
  int n;
  float lr, b1, b2, eps, c1, c2;
  AdamTensor t[2 * MLP_MAX_LAYERS];
};

__device__ __forceinline__ float adamw_update(float& w, float g, float& m, float& v, float lr, float b1, float b2,
                                              float eps, float wd, float c1, float c2) {
  m = b1 * m + (1.f - b1) * g;
  v = b2 * v + (1.f - b2) * g * g;
  float wi = w * (1.f - lr * wd);
  wi -= lr * (m / c1) / (sqrtf(v / c2) + eps);
  w = wi;
  return wi;
}

__global__ void __launch_bounds__(256) adamw_multi_kernel(const __grid_constant__ AdamJobs j) {
  __shared__ float tile[32][33];
  int q = 0;
  while (q + 1 < j.n && (int)blockIdx.x >= j.t[q + 1].first) ++q;
  const AdamTensor& t = j.t[q];
  const int tiles_c = (t.cols + 31) / 32, b = (int)blockIdx.x - t.first;
  const int r0 = b / tiles_c * 32, c0 = b % tiles_c * 32;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    const int r = r0 + y + i, c = c0 + x;
    if (r < t.rows && c < t.cols) {
      const size_t e = (size_t)r * t.cols + c;
      float w = t.w[e], m = t.m[e], v = t.v[e];
      adamw_update(w, t.g[e], m, v, j.lr, j.b1, j.b2, j.eps, t.wd, j.c1, j.c2);
      t.w[e] = w;
      t.m[e] = m;
      t.v[e] = v;
      if (t.wb) t.wb[(size_t)r * t.ldw + c] = __float2bfloat16(w);
      tile[y + i][x] = w;
    }
  }
  if (!t.wt) return;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    const int c = c0 + y + i, r = r0 + x;
    if (c < t.cols && r < t.rows) t.wt[(size_t)c * t.ldt + r] = __float2bfloat16(tile[x][y + i]);
  }
}

// mean-squared-error gradient dY = 2 (Y - T) / (R C) (FP32, and bf16 with row
// stride ldb); loss partial sums accumulated into *loss, one atomic per CTA
__global__ void __launch_bounds__(256)
    mse_grad_kernel(const float* __restrict__ y, const float* __restrict__ t, float* __restrict__ gf,
                    __nv_bfloat16* __restrict__ gb, int rows, int cols, int ldb, float scale, double* loss) {
  __shared__ double part[8];
  double acc = 0.0;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
      const size_t i = (size_t)r * cols + c;
      const float d = y[i] - t[i];
      acc += (double)d * d;
      const float g = 2.f * d * scale;
      gf[i] = g;
      gb[(size_t)r * ldb + c] = __float2bfloat16(g);
    }
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) acc += part[w];
    atomicAdd(loss, acc);
  }
}

// AdamW on FP32 master weights; refreshes the bf16 copy
__global__ void adamw_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                             float* __restrict__ v, __nv_bfloat16* __restrict__ wb, long long n, float lr, float b1,
                             float b2, float eps, float wd, float c1, float c2) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float wi = adamw_update(w[i], g[i], m[i], v[i], lr, b1, b2, eps, wd, c1, c2);
    if (wb) wb[i] = __float2bfloat16(wi);
  }
}

// y[b][c * nsteps + t] += Bloch component c at time (t + 1) dt of the system
// without the bath: precession of (0, 0, 1) about (Omega, 0, eps) at angular
// frequency w = sqrt(Omega^2 + eps^2) (Rodrigues' rotation).
__global__ void bloch_free_add_kernel(float* __restrict__ y, const float* __restrict__ oe, int B, int nsteps,
                                      float dt) {
  const long long total = (long long)B * nsteps;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int b = (int)(i / nsteps), t = (int)(i - (long long)b * nsteps);
    const float om = oe[2 * b], ep = oe[2 * b + 1];
    const float w = sqrtf(om * om + ep * ep);
    const float nx = w > 0.f ? om / w : 0.f, nz = w > 0.f ? ep / w : 1.f;
    float s, c;
    sincosf(w * dt * (float)(t + 1), &s, &c);
    float* row = y + (size_t)b * 3 * nsteps;
    row[t] += nx * nz * (1.f - c);
    row[nsteps + t] += -nx * s;
    row[2 * nsteps + t] += c + nz * nz * (1.f - c);
  }
}

}  // namespace otb

using namespace otb;

namespace {

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder (null where the driver has none).
EncodeTiled tensor_map_encoder() {
  static EncodeTiled f = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return (EncodeTiled)p;
  }();
  return f;
}

// Map of an operand of `rows` logical rows and depth K: stored [rows][K] (box
// 64 x box_rows) or, transposed, [K][rows] (box 64 x 64); ld elements per
// stored row, a multiple of 8.
bool operand_map(CUtensorMap* map, const void* p, int rows, int K, int ld, bool trans, int box_rows) {
  EncodeTiled enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)(trans ? rows : K), (cuuint64_t)(trans ? K : rows)};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)(trans ? 64 : box_rows)};
  const cuuint32_t ones[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, ones,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
otb_status launch_tma(const void* A, int lda, bool ta, const void* B, int ldb, bool tb, int M, int N, int K,
                      const GemmOut& out, int sms, int32_t* err, cudaStream_t stream) {
  CUtensorMap ma, mb;
  if (!operand_map(&ma, A, M, K, lda, ta, TM_BM) || !operand_map(&mb, B, N, K, ldb, tb, BN))
    return set_error(OTB_ERR_CUDA, "tensor map");
  const int tiles = ((M + TM_BM - 1) / TM_BM) * ((N + BN - 1) / BN);
  if (!check_cuda(cudaFuncSetAttribute(tc_gemm_tma_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       TmShape<BN>::smem),
                  "tma gemm smem"))
    return OTB_ERR_CUDA;
  tc_gemm_tma_kernel<BN><<<std::min(tiles, sms), TM_THREADS, TmShape<BN>::smem, stream>>>(ma, mb, M, N, K, ta, tb, out,
                                                                                          err);
  if (!check_cuda(cudaGetLastError(), "tma gemm")) return OTB_ERR_CUDA;
  return OTB_OK;
}

// a few rows per CTA, four CTAs per SM
void launch_mse(const float* y, const float* t, float* gf, __nv_bfloat16* gb, int rows, int cols, int ldb, float scale,
                double* loss, cudaStream_t s) {
  mse_grad_kernel<<<std::min(rows, 608), 256, 0, s>>>(y, t, gf, gb, rows, cols, ldb, scale, loss);
}

bool tma_operand(const void* p, int ld) { return ld % 8 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Out = A B^T, A [M][K] (lda; transposed: [K][M]) and B [N][K] (ldb; transposed:
// [K][N]) with 16-byte aligned rows.
otb_status gemm_tma(const void* A, int lda, bool ta, const void* B, int ldb, bool tb, int M, int N, int K,
                    const GemmOut& out, int32_t* err, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  sms = std::max(sms, 1);
  const int mt = (M + TM_BM - 1) / TM_BM;
  if (mt * ((N + 255) / 256) >= sms) return launch_tma<256>(A, lda, ta, B, ldb, tb, M, N, K, out, sms, err, stream);
  if (mt * ((N + 127) / 128) >= sms) return launch_tma<128>(A, lda, ta, B, ldb, tb, M, N, K, out, sms, err, stream);
  return launch_tma<64>(A, lda, ta, B, ldb, tb, M, N, K, out, sms, err, stream);
}

}  // namespace

extern "C" otb_status otb_mlp_gemm(const void* A, const void* B, int32_t M, int32_t N, int32_t K,
                                   const float* bias, int32_t epilogue, const float* z_in, float* z_out,
                                   float* out_f32, void* out_bf16, int32_t* err, void* stream) {
  if (!A || !B || !err || M <= 0 || N <= 0 || K <= 0 || epilogue < 0 || epilogue > 2)
    return set_error(OTB_ERR_INVALID_ARG, "bad gemm arguments");
  if (epilogue == EPI_GELU_GRAD && !z_in) return set_error(OTB_ERR_INVALID_ARG, "gelu-grad needs z_in");
  if (tma_operand(A, K) && tma_operand(B, K) && tensor_map_encoder()) {
    const GemmOut out{bias, z_in, z_out, out_f32, (__nv_bfloat16*)out_bf16, N, N, epilogue};
    return gemm_tma(A, K, false, B, K, false, M, N, K, out, err, (cudaStream_t)stream);
  }
  dim3 grid((N + TC_BN - 1) / TC_BN, (M + TC_BM - 1) / TC_BM);
  constexpr int smem = 2 * (TC_BM + TC_BN) * TC_BK * 2;   // two A + B stages, 64 KiB
  if (!check_cuda(cudaFuncSetAttribute(tc_gemm_pipe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                  "tc gemm smem"))
    return OTB_ERR_CUDA;
  tc_gemm_pipe_kernel<<<grid, TC_THREADS, smem, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)A, (const __nv_bfloat16*)B, M, N, K, bias, epilogue, z_in, z_out, out_f32,
      (__nv_bfloat16*)out_bf16, err);
  if (!check_cuda(cudaGetLastError(), "tc gemm")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_transpose_bf16(const void* in, void* out, int32_t R, int32_t C, void* stream) {
  if (!in || !out || R <= 0 || C <= 0) return set_error(OTB_ERR_INVALID_ARG, "bad transpose arguments");
  dim3 grid((C + 31) / 32, (R + 31) / 32), block(32, 8);
  transpose_bf16_kernel<<<grid, block, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out,
                                                                  R, C);
  if (!check_cuda(cudaGetLastError(), "transpose")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_f32_to_bf16(const float* in, void* out, int64_t n, void* stream) {
  if (!in || !out || n < 0) return set_error(OTB_ERR_INVALID_ARG, "bad conversion arguments");
  if (n == 0) return OTB_OK;
  f32_to_bf16_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>(in, (__nv_bfloat16*)out, n);
  if (!check_cuda(cudaGetLastError(), "f32->bf16")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_colsum(const float* in, float* out, int32_t R, int32_t C, void* stream) {
  if (!in || !out || R <= 0 || C <= 0) return set_error(OTB_ERR_INVALID_ARG, "bad colsum arguments");
  colsum_kernel<<<(C + 127) / 128, 128, 0, (cudaStream_t)stream>>>(in, out, R, C);
  if (!check_cuda(cudaGetLastError(), "colsum")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_mse_grad(const float* y, const float* t, float* g_f32, void* g_bf16, int64_t n,
                                       double* loss, void* stream) {
  if (!y || !t || !g_f32 || !g_bf16 || !loss || n <= 0) return set_error(OTB_ERR_INVALID_ARG, "bad mse arguments");
  // flat: rows of 1024 values and a remainder row
  const int64_t rows = n / 1024, rest = n % 1024;
  if (rows > INT32_MAX) return set_error(OTB_ERR_INVALID_ARG, "bad mse arguments");
  cudaStream_t s = (cudaStream_t)stream;
  __nv_bfloat16* gb = (__nv_bfloat16*)g_bf16;
  if (rows) launch_mse(y, t, g_f32, gb, (int)rows, 1024, 1024, 1.f / (float)n, loss, s);
  if (rest) {
    const int64_t o = rows * 1024;
    launch_mse(y + o, t + o, g_f32 + o, gb + o, 1, (int)rest, (int)rest, 1.f / (float)n, loss, s);
  }
  if (!check_cuda(cudaGetLastError(), "mse")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_mse_grad_rows(const float* y, const float* t, float* g_f32, void* g_bf16, int32_t rows,
                                            int32_t cols, int32_t ld_bf16, double* loss, void* stream) {
  if (!y || !t || !g_f32 || !g_bf16 || !loss || rows <= 0 || cols <= 0 || ld_bf16 < cols)
    return set_error(OTB_ERR_INVALID_ARG, "bad mse arguments");
  launch_mse(y, t, g_f32, (__nv_bfloat16*)g_bf16, rows, cols, ld_bf16, 1.f / (float)((int64_t)rows * cols), loss,
             (cudaStream_t)stream);
  if (!check_cuda(cudaGetLastError(), "mse")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_gemm_strided(const void* A, int32_t lda, int32_t trans_a, const void* B, int32_t ldb,
                                           int32_t trans_b, int32_t M, int32_t N, int32_t K, const float* bias,
                                           int32_t epilogue, const float* z_in, float* z_out, float* out_f32,
                                           void* out_bf16, int32_t ld_bf16, int32_t* err, void* stream) {
  if (!A || !B || !err || M <= 0 || N <= 0 || K <= 0 || epilogue < 0 || epilogue > 2 ||
      lda < (trans_a ? M : K) || ldb < (trans_b ? N : K) || (out_bf16 && ld_bf16 < N))
    return set_error(OTB_ERR_INVALID_ARG, "bad gemm arguments");
  if (epilogue == EPI_GELU_GRAD && !z_in) return set_error(OTB_ERR_INVALID_ARG, "gelu-grad needs z_in");
  if (!tma_operand(A, lda) || !tma_operand(B, ldb))
    return set_error(OTB_ERR_INVALID_ARG, "operand rows must be 16-byte aligned");
  const GemmOut out{bias, z_in, z_out, out_f32, (__nv_bfloat16*)out_bf16, N, out_bf16 ? ld_bf16 : N, epilogue};
  return gemm_tma(A, lda, trans_a != 0, B, ldb, trans_b != 0, M, N, K, out, err, (cudaStream_t)stream);
}

extern "C" otb_status otb_mlp_colsums(int32_t n, const float* const* in, float* const* out, int32_t rows,
                                      const int32_t* cols, void* stream) {
  if (n < 1 || n > MLP_MAX_LAYERS || !in || !out || !cols || rows <= 0)
    return set_error(OTB_ERR_INVALID_ARG, "bad colsum arguments");
  ColsumJobs j;
  j.n = n;
  j.rows = rows;
  int first = 0;
  for (int i = 0; i < n; ++i) {
    if (!in[i] || !out[i] || cols[i] <= 0) return set_error(OTB_ERR_INVALID_ARG, "bad colsum arguments");
    j.first[i] = first;
    j.cols[i] = cols[i];
    j.in[i] = in[i];
    j.out[i] = out[i];
    first += (cols[i] + 31) / 32;
  }
  j.first[n] = first;
  colsum_multi_kernel<<<first, 256, 0, (cudaStream_t)stream>>>(j);
  if (!check_cuda(cudaGetLastError(), "colsums")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_adamw_net(int32_t n, const otb_mlp_layer* layers, float lr, float beta1, float beta2,
                                        float eps, float weight_decay, int32_t step, void* stream) {
  if (n < 1 || n > MLP_MAX_LAYERS || !layers || step < 1) return set_error(OTB_ERR_INVALID_ARG, "bad adamw arguments");
  AdamJobs j;
  j.n = 2 * n;
  j.lr = lr;
  j.b1 = beta1;
  j.b2 = beta2;
  j.eps = eps;
  j.c1 = 1.f - powf(beta1, (float)step);
  j.c2 = 1.f - powf(beta2, (float)step);
  int first = 0;
  for (int i = 0; i < n; ++i) {
    const otb_mlp_layer& l = layers[i];
    if (l.fout <= 0 || l.fin <= 0 || !l.w || !l.gw || !l.mw || !l.vw || !l.b || !l.gb || !l.mb || !l.vb || !l.w_bf16 ||
        !l.wt_bf16 || l.ld_w < l.fin || l.ld_wt < l.fout)
      return set_error(OTB_ERR_INVALID_ARG, "bad adamw arguments");
    j.t[2 * i] = AdamTensor{l.w, l.mw, l.vw, l.gw, (__nv_bfloat16*)l.w_bf16, (__nv_bfloat16*)l.wt_bf16,
                            l.fout, l.fin, l.ld_w, l.ld_wt, first, weight_decay};
    first += ((l.fout + 31) / 32) * ((l.fin + 31) / 32);
    j.t[2 * i + 1] = AdamTensor{l.b, l.mb, l.vb, l.gb, nullptr, nullptr, 1, l.fout, 0, 0, first, 0.f};
    first += (l.fout + 31) / 32;
  }
  adamw_multi_kernel<<<first, 256, 0, (cudaStream_t)stream>>>(j);
  if (!check_cuda(cudaGetLastError(), "adamw")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_adamw(float* w, const float* g, float* m, float* v, void* w_bf16, int64_t n, float lr,
                                    float beta1, float beta2, float eps, float weight_decay, int32_t step,
                                    void* stream) {
  if (!w || !g || !m || !v || n <= 0 || step < 1) return set_error(OTB_ERR_INVALID_ARG, "bad adamw arguments");
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  adamw_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>(w, g, m, v, (__nv_bfloat16*)w_bf16, n, lr, beta1, beta2, eps,
                                                       weight_decay, c1, c2);
  if (!check_cuda(cudaGetLastError(), "adamw")) return OTB_ERR_CUDA;
  return OTB_OK;
}

extern "C" otb_status otb_mlp_bloch_free_add(float* y, const float* omega_eps, int32_t B, int32_t nsteps, float dt,
                                            void* stream) {
  if (!y || !omega_eps || B <= 0 || nsteps <= 0 || !(dt > 0.f))
    return set_error(OTB_ERR_INVALID_ARG, "bad bloch arguments");
  bloch_free_add_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>(y, omega_eps, B, nsteps, dt);
  if (!check_cuda(cudaGetLastError(), "bloch free add")) return OTB_ERR_CUDA;
  return OTB_OK;
}
