// BF16 x BF16 -> FP32 GEMM on the 5th-generation tensor cores (sm_103a).
//
//   C[M x N] = A[M x K] * B[N x K]^T        (both operands K-major, row-major)
//
// One CTA computes a 128 x BN tile.  Thread 0 streams 128x64 tiles of A and
// BNx64 tiles of B into shared memory with TMA (128-byte swizzle), issues
// tcgen05.mma (M = 128, N = BN, K = 16 per instruction) into a TMEM
// accumulator, and releases each stage with tcgen05.commit on the stage's
// "empty" mbarrier.  After the last commit the four warps read the
// accumulator back with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31, i.e.
// rows 32w..32w+31 of the tile).
//
// Every mbarrier wait is bounded; a wait that runs out sets *err, the CTA
// waits (bounded) for the copies it issued, frees its TMEM and returns.
//
// k_gemm_tn is the plain product; the surrogate's training passes (k_train_*)
// and its inference (k_mlp_ensemble) build on the same pieces.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "internal.h"

namespace cacg {
namespace gemm {

namespace {

constexpr int BM = 128, BK = 64, NT = 128;
constexpr unsigned WAIT_LIMIT = 1u << 26;

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait: false when the limit ran out
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  for (unsigned it = 0; it < WAIT_LIMIT; it++)
    if (mbar_try(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap *map, int x, int y,
                                            unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// K-major operand, 128-byte swizzle: 8-row atoms of 128 B, 1024 B apart
__device__ __forceinline__ unsigned long long sw128_desc(unsigned addr) {
  unsigned long long d = 0;
  d |= (unsigned long long) ((addr >> 4) & 0x3FFF);
  d |= (unsigned long long) 1 << 16;                  // leading byte offset (unused)
  d |= (unsigned long long) (1024 >> 4) << 32;        // stride byte offset
  d |= (unsigned long long) 1 << 46;                  // descriptor version
  d |= (unsigned long long) 2 << 61;                  // 128-byte swizzle
  return d;
}

// kind::f16 instruction descriptor: D f32, A/B bf16, both K-major, M = 128
__host__ __device__ constexpr unsigned idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned) (n >> 3) << 17) |
         ((unsigned) (BM >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(unsigned tmem, unsigned long long a, unsigned long long b,
                                         unsigned idesc, unsigned acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void mma_commit(unsigned bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// sigma(z) = (1 + tanh(z / 2)) / 2 and silu(z) = z sigma(z) = h + h tanh(h), h = z / 2, on
// the hardware tanh (tanh.approx.f32: one special-function instruction against two for
// exp and reciprocal; its error, about 2^-11, is below the bf16 rounding of the
// activations, 2^-9)
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sigmoidf_(float z) { return fmaf(0.5f, tanh_approx(0.5f * z), 0.5f); }
__device__ __forceinline__ float siluf_(float z) {
  const float h = 0.5f * z;
  return fmaf(h, tanh_approx(h), h);
}

struct Epi {
  float *c;
  int ldc;
};

template <int BN, int STAGES>
__global__ void __launch_bounds__(NT, 1)
k_gemm_tn(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
          int M, int N, int K, Epi ep, int *err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // stage buffers on a 1024-byte boundary (swizzle atoms)
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
  constexpr int TMEM_COLS = BN < 32 ? 32 : BN;
  unsigned char *sa = base;
  unsigned char *sb = base + STAGES * A_BYTES;
  unsigned long long *bars =
      reinterpret_cast<unsigned long long *>(sb + STAGES * B_BYTES);  // full, empty, done
  unsigned *tmem_slot = reinterpret_cast<unsigned *>(bars + 2 * STAGES + 1);
  __shared__ int s_fail;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int nk = K / BK;

  if (threadIdx.x == 0) {
    s_fail = 0;
    for (int i = 0; i < 2 * STAGES + 1; i++) mbar_init(smem_u32(bars + i), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;

  if (threadIdx.x == 0) {
    const unsigned idesc = idesc_bf16(BN);
    int issued = 0, consumed = 0;
    bool ok = true;
    for (int s = 0; s < STAGES && s < nk; s++) {
      unsigned fb = smem_u32(bars + s);
      mbar_expect_tx(fb, A_BYTES + B_BYTES);
      tma_load_2d(smem_u32(sa + s * A_BYTES), &tma_a, s * BK, m0, fb);
      tma_load_2d(smem_u32(sb + s * B_BYTES), &tma_b, s * BK, n0, fb);
      issued++;
    }
    for (int kt = 0; kt < nk && ok; kt++) {
      const int s = kt % STAGES;
      const unsigned par = (kt / STAGES) & 1;
      if (!mbar_wait(smem_u32(bars + s), par)) {
        ok = false;
        break;
      }
      consumed++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned a_addr = smem_u32(sa + s * A_BYTES), b_addr = smem_u32(sb + s * B_BYTES);
#pragma unroll
      for (int kk = 0; kk < BK / 16; kk++)
        mma_bf16(tmem, sw128_desc(a_addr + kk * 32), sw128_desc(b_addr + kk * 32), idesc,
                 (kt | kk) != 0);
      mma_commit(smem_u32(bars + STAGES + s));
      // refill the stage the previous k-tile used, once its MMAs are done
      if (kt >= 1) {
        const int pk = kt - 1, ps = pk % STAGES, nxt = pk + STAGES;
        if (nxt < nk) {
          if (!mbar_wait(smem_u32(bars + STAGES + ps), (pk / STAGES) & 1)) {
            ok = false;
            break;
          }
          unsigned fb = smem_u32(bars + ps);
          mbar_expect_tx(fb, A_BYTES + B_BYTES);
          tma_load_2d(smem_u32(sa + ps * A_BYTES), &tma_a, nxt * BK, m0, fb);
          tma_load_2d(smem_u32(sb + ps * B_BYTES), &tma_b, nxt * BK, n0, fb);
          issued++;
        }
      }
    }
    if (ok) {
      mma_commit(smem_u32(bars + 2 * STAGES));
    } else {
      atomicExch(err, 1);
      // let the copies and MMAs already issued finish before the CTA's
      // shared memory and TMEM go away
      for (int k = consumed; k < issued; k++) mbar_wait(smem_u32(bars + k % STAGES), (k / STAGES) & 1);
      mma_commit(smem_u32(bars + 2 * STAGES));
      mbar_wait(smem_u32(bars + 2 * STAGES), 0);
      s_fail = 1;
    }
  }
  __syncwarp();
  // all threads: wait for the accumulator (or the failure flag)
  bool ready = false;
  for (unsigned it = 0; it < WAIT_LIMIT; it++) {
    if (mbar_try(smem_u32(bars + 2 * STAGES), 0)) {
      ready = true;
      break;
    }
    if (*((volatile int *) &s_fail)) break;
  }
  if (!ready && threadIdx.x == 0) atomicExch(err, 2);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  if (__all_sync(0xffffffffu, ready ? 1 : 0)) {
    const int row = m0 + warp * 32 + lane;
    const unsigned tl = tmem + ((unsigned) (warp * 32) << 16);
#pragma unroll 1
    for (int c = 0; c < BN; c += 16) {
      float v[16];
      tmem_ld16(tl + c, v);
      if (row >= M) continue;
      const int col = n0 + c;
      const bool full = col + 16 <= N;
      float *dst = ep.c + (size_t) row * ep.ldc + col;
      if (full && (ep.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++)
          reinterpret_cast<float4 *>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; i++)
          if (col + i < N) dst[i] = v[i];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TMEM_COLS)
                 : "memory");
  }
}

// ---------------------------------------------------------------- fused ensemble
//
// The whole surrogate ensemble for 128 elements per CTA in one launch:
// for each member k and layer l the CTA runs D = A_l W_l^T on the tensor cores
// (A_1 = the features tile sX, A_l = the previous layer's activations in sA),
// reads D back from TMEM, applies bias + SiLU and writes the BF16 activations
// into sA in the same 128-byte-swizzled K-major layout TMA would produce, so
// the next layer's MMAs read them directly.  The 13 weight k-tiles of each
// member (W1: 1, W2: 4, W3: 4, W4: 4) stream through four shared-memory
// stages, loaded by TMA up to four tiles ahead of the MMAs.  Sixteen warps
// share the epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (its rows)
// and columns 64 (w / 4) .. + 63.  The last layer's
// outputs are summed over the members in registers; the kernel writes the
// denormalised ensemble mean and the spread (largest per-output standard
// deviation across members).
constexpr int ENS_NT = 512, ENS_STAGES = 4, ENS_H = 256, ENS_OUT = 24, ENS_BSTRIDE = 3 * 256 + 24;
constexpr int ENS_MAX_MEMBERS = 4;  // shared memory: 16 + 64 + 4 x 32 KB + biases
constexpr int ENS_X_BYTES = BM * BK * 2, ENS_A_BYTES = BM * ENS_H * 2, ENS_W_BYTES = ENS_H * BK * 2;

struct EnsArgs {
  const float *bias;  // [members][b1 256, b2 256, b3 256, b4 24]
  const float *norm;  // out_mean at [64, 88), out_std at [88, 112)
  float *mean, *spread;
  int n, members;
  int *err;
  const int *count;  // rows to evaluate (device; null: n); CTAs past it return at once
};

__device__ __forceinline__ void ens_issue(int g, const CUtensorMap *w1, const CUtensorMap *w2,
                                          const CUtensorMap *w3, const CUtensorMap *w4,
                                          unsigned char *sw, unsigned long long *full) {
  const int k = g / 13, r = g % 13;
  const int st = g % ENS_STAGES;
  const unsigned fb = smem_u32(full + st), dst = smem_u32(sw + st * ENS_W_BYTES);
  if (r == 0) {
    mbar_expect_tx(fb, ENS_W_BYTES);
    tma_load_2d(dst, w1, 0, k * ENS_H, fb);
  } else if (r < 5) {
    mbar_expect_tx(fb, ENS_W_BYTES);
    tma_load_2d(dst, w2, (r - 1) * BK, k * ENS_H, fb);
  } else if (r < 9) {
    mbar_expect_tx(fb, ENS_W_BYTES);
    tma_load_2d(dst, w3, (r - 5) * BK, k * ENS_H, fb);
  } else {
    mbar_expect_tx(fb, 32 * BK * 2);
    tma_load_2d(dst, w4, (r - 9) * BK, k * ENS_OUT, fb);
  }
}

// byte offset of (row, 16-byte chunk) in a 128-row, 64-column bf16 SW128 atom column
__device__ __forceinline__ unsigned sw128_off(int row, int chunk) {
  return (unsigned) ((row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4));
}

__global__ void __launch_bounds__(ENS_NT, 1)
k_mlp_ensemble(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w1,
               const __grid_constant__ CUtensorMap tma_w2, const __grid_constant__ CUtensorMap tma_w3,
               const __grid_constant__ CUtensorMap tma_w4, EnsArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const int nrows = a.count ? *a.count : a.n;
  if ((int) blockIdx.x * BM >= nrows) return;  // before any barrier or allocation
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  unsigned char *sx = base;
  unsigned char *sa = sx + ENS_X_BYTES;
  unsigned char *sw = sa + ENS_A_BYTES;
  float *sbias = reinterpret_cast<float *>(sw + ENS_STAGES * ENS_W_BYTES);
  unsigned long long *bars =
      reinterpret_cast<unsigned long long *>(sbias + a.members * ENS_BSTRIDE);  // full[3] empty[3] x done
  unsigned *tmem_slot = reinterpret_cast<unsigned *>(bars + 2 * ENS_STAGES + 2);
  unsigned long long *full = bars, *empty = bars + ENS_STAGES, *xbar = bars + 2 * ENS_STAGES,
                     *done = bars + 2 * ENS_STAGES + 1;
  __shared__ int s_fail;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wg = warp >> 2, q = warp & 3, row = q * 32 + lane;
  const int m0 = blockIdx.x * BM;
  const int T = 13 * a.members;

  for (int i = tid; i < a.members * ENS_BSTRIDE; i += ENS_NT) sbias[i] = a.bias[i];
  if (tid == 0) {
    s_fail = 0;
    for (int i = 0; i < 2 * ENS_STAGES + 2; i++) mbar_init(smem_u32(bars + i), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(ENS_H)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;

  int issued = 0;
  if (tid == 0) {
    mbar_expect_tx(smem_u32(xbar), ENS_X_BYTES);
    tma_load_2d(smem_u32(sx), &tma_x, 0, m0, smem_u32(xbar));
    for (; issued < ENS_STAGES && issued < T; issued++)
      ens_issue(issued, &tma_w1, &tma_w2, &tma_w3, &tma_w4, sw, full);
  }
  float s1[ENS_OUT], s2[ENS_OUT];
#pragma unroll
  for (int c = 0; c < ENS_OUT; c++) s1[c] = s2[c] = 0.f;

  int g = 0;        // next weight tile to consume
  int nlayer = 0;   // layers completed (parity of `done`)
  bool ok = true;
  for (int k = 0; k < a.members && ok; k++) {
    const float *bk = sbias + k * ENS_BSTRIDE;
    for (int l = 1; l <= 4 && ok; l++) {
      if (tid == 0) {
        bool good = true;
        if (g == 0) good = mbar_wait(smem_u32(xbar), 0);
        const int nk = l == 1 ? 1 : 4;
        const unsigned idesc = idesc_bf16(l == 4 ? 32 : ENS_H);
        for (int kt = 0; kt < nk && good; kt++, g++) {
          const int st = g % ENS_STAGES;
          if (!mbar_wait(smem_u32(full + st), (g / ENS_STAGES) & 1)) {
            good = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned a_addr = l == 1 ? smem_u32(sx) : smem_u32(sa + kt * (BM * BK * 2));
          const unsigned b_addr = smem_u32(sw + st * ENS_W_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / 16; kk++)
            mma_bf16(tmem, sw128_desc(a_addr + kk * 32), sw128_desc(b_addr + kk * 32), idesc,
                     (kt | kk) != 0);
          mma_commit(smem_u32(empty + st));
          if (g >= 1 && issued < T) {  // refill the stage the previous tile used
            const int pg = g - 1;
            if (!mbar_wait(smem_u32(empty + pg % ENS_STAGES), (pg / ENS_STAGES) & 1)) {
              good = false;
              break;
            }
            ens_issue(issued++, &tma_w1, &tma_w2, &tma_w3, &tma_w4, sw, full);
          }
        }
        mma_commit(smem_u32(done));
        if (!good) {
          atomicExch(a.err, 1);
          s_fail = 1;
        }
      }
      __syncwarp();
      bool ready = false;
      for (unsigned it = 0; it < WAIT_LIMIT; it++) {
        if (mbar_try(smem_u32(done), nlayer & 1)) {
          ready = true;
          break;
        }
      }
      nlayer++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned tl = tmem + ((unsigned) (q * 32) << 16);
      if (l < 4) {
        const float *b = bk + (l - 1) * ENS_H;
#pragma unroll 1
        for (int c = wg * 64; c < wg * 64 + 64; c += 16) {
          float v[16];
          tmem_ld16(tl + c, v);
          unsigned w[8];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            float z0 = v[2 * i] + b[c + 2 * i], z1 = v[2 * i + 1] + b[c + 2 * i + 1];
            __nv_bfloat162 h2 = __floats2bfloat162_rn(siluf_(z0), siluf_(z1));
            w[i] = *reinterpret_cast<unsigned *>(&h2);
          }
          const int ac = c >> 6, ch = (c & 63) >> 3;
          unsigned char *dst = sa + ac * (BM * BK * 2);
          *reinterpret_cast<uint4 *>(dst + sw128_off(row, ch)) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4 *>(dst + sw128_off(row, ch + 1)) = make_uint4(w[4], w[5], w[6], w[7]);
        }
      } else if (wg == 0) {
        const float *b = bk + 3 * ENS_H;
        float v0[16], v1[16];
        tmem_ld16(tl, v0);
        tmem_ld16(tl + 16, v1);
#pragma unroll
        for (int c = 0; c < ENS_OUT; c++) {
          float y = (c < 16 ? v0[c] : v1[c - 16]) + b[c];
          s1[c] += y;
          s2[c] += y * y;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (__syncthreads_or(!ready || *((volatile int *) &s_fail))) ok = false;
    }
  }
  if (!ok && tid == 0) {
    atomicExch(a.err, 2);
    // let the weight copies already issued land before the CTA exits
    for (int t = g; t < issued; t++) mbar_wait(smem_u32(full + t % ENS_STAGES), (t / ENS_STAGES) & 1);
  }
  if (ok && wg == 0 && m0 + row < nrows) {
    const float inv = 1.f / a.members;
    float smax = 0.f;
    float *mo = a.mean + (size_t) (m0 + row) * ENS_OUT;
#pragma unroll
    for (int c = 0; c < ENS_OUT; c++) {
      const float mu = s1[c] * inv, var = fmaxf(s2[c] * inv - mu * mu, 0.f);
      const float sd = a.norm[88 + c];
      mo[c] = mu * sd + a.norm[64 + c];
      smax = fmaxf(smax, sqrtf(var) * sd);
    }
    a.spread[m0 + row] = smax;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ENS_H)
                 : "memory");
  }
}

// ---------------------------------------------------------------- training
//
// One Adam step of every member at once: grid.y (or .x) runs over the members,
// whose activations, weights and gradients are stacked.  A layer kernel forms a
// 128-row tile of one layer (forward or backward) and writes what the next
// kernels read, as they read it: the activation (or gradient) row-major, K-major
// for the next layer, and transposed, K-major for the weight gradients, so that
// no transpose runs by itself; Z transposed within the tile, so that a warp's
// loads and stores are whole lines.  The weight gradients of all layers are one
// launch; the update kernel adds up the bias gradients in a fixed order (no
// atomics: the same result at every run) and does Adam and the new BF16 weights.
//
// What bounded it: launches and idle SMs.  One member's 2,048-row step was 45
// launches, GEMMs on 2 to 16 blocks whose epilogues stored one float a line,
// and took 508 us; the step of four members now takes 10 launches.
constexpr int TR_NT = 512, TR_STAGES = 4, TR_A = BM * BK * 2, TR_B = 256 * BK * 2;
constexpr int TR_H = 256, TR_IN = 64, TR_OUT = 24, TR_OUTP = 64;

size_t train_smem() { return 1024 + (size_t) TR_STAGES * (TR_A + TR_B) + (2 * TR_STAGES + 1) * 8 + 16; }

struct TrainSmem {
  unsigned char *sa, *sb;
  unsigned long long *bars;  // full, empty, done
  unsigned *tmem_slot;
};

__device__ __forceinline__ TrainSmem train_smem_of(unsigned char *raw) {
  TrainSmem m;
  m.sa = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) &
                                           ~static_cast<uintptr_t>(1023));
  m.sb = m.sa + TR_STAGES * TR_A;
  m.bars = reinterpret_cast<unsigned long long *>(m.sb + TR_STAGES * TR_B);
  m.tmem_slot = reinterpret_cast<unsigned *>(m.bars + 2 * TR_STAGES + 1);
  return m;
}

// barriers and a 256-column TMEM accumulator; all threads
__device__ __forceinline__ unsigned train_begin(const TrainSmem &m, int *s_fail) {
  if (threadIdx.x == 0) {
    *s_fail = 0;
    for (int i = 0; i < 2 * TR_STAGES + 1; i++) mbar_init(smem_u32(m.bars + i), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(m.tmem_slot)),
                 "r"(256)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return *m.tmem_slot;
}

__device__ __forceinline__ void train_end(unsigned tmem) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
  }
}

// D[128][bn] = sum over nk k-tiles of A rows ya.. and B rows yb..;
// thread 0 streams and issues, all threads wait: true when D is complete
__device__ __forceinline__ bool train_mma(const TrainSmem &m, unsigned tmem, const CUtensorMap *ta,
                                          const CUtensorMap *tb, int nk, int ya, int yb,
                                          int bn, int *err, int *s_fail) {
  if (threadIdx.x == 0) {
    const unsigned idesc = idesc_bf16(bn), bytes = TR_A + (unsigned) bn * BK * 2;
    int issued = 0, consumed = 0;
    bool ok = true;
    auto load = [&](int kt) {
      const int st = kt % TR_STAGES;
      const unsigned fb = smem_u32(m.bars + st);
      mbar_expect_tx(fb, bytes);
      tma_load_2d(smem_u32(m.sa + st * TR_A), ta, kt * BK, ya, fb);
      tma_load_2d(smem_u32(m.sb + st * TR_B), tb, kt * BK, yb, fb);
      issued++;
    };
    for (int kt = 0; kt < TR_STAGES && kt < nk; kt++) load(kt);
    for (int kt = 0; kt < nk && ok; kt++) {
      const int st = kt % TR_STAGES;
      if (!mbar_wait(smem_u32(m.bars + st), (kt / TR_STAGES) & 1)) {
        ok = false;
        break;
      }
      consumed++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned a_addr = smem_u32(m.sa + st * TR_A), b_addr = smem_u32(m.sb + st * TR_B);
#pragma unroll
      for (int kk = 0; kk < BK / 16; kk++)
        mma_bf16(tmem, sw128_desc(a_addr + kk * 32), sw128_desc(b_addr + kk * 32), idesc,
                 (kt | kk) != 0);
      mma_commit(smem_u32(m.bars + TR_STAGES + st));
      // refill the stage the previous k-tile used, once its MMAs are done
      if (kt >= 1 && kt - 1 + TR_STAGES < nk) {
        const int pk = kt - 1, ps = pk % TR_STAGES;
        if (!mbar_wait(smem_u32(m.bars + TR_STAGES + ps), (pk / TR_STAGES) & 1)) {
          ok = false;
          break;
        }
        load(pk + TR_STAGES);
      }
    }
    mma_commit(smem_u32(m.bars + 2 * TR_STAGES));
    if (!ok) {
      atomicExch(err, 1);
      // let the copies and MMAs already issued finish before the block's shared
      // memory and TMEM go away
      for (int k = consumed; k < issued; k++)
        mbar_wait(smem_u32(m.bars + k % TR_STAGES), (k / TR_STAGES) & 1);
      mbar_wait(smem_u32(m.bars + 2 * TR_STAGES), 0);
      *s_fail = 1;
    }
  }
  __syncwarp();
  const bool ready = mbar_wait(smem_u32(m.bars + 2 * TR_STAGES), 0);
  if (!ready && (threadIdx.x & 31) == 0) atomicExch(err, 2);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return __syncthreads_and(ready && *((volatile int *) s_fail) == 0) != 0;
}

struct TrainLayer {
  int B, nk, bn, brows;        // rows per member, k-tiles, tile width, weight rows per member
  const float *bias;           // member m's at bias + m * pstride
  long pstride;
  float *z;                    // [tile][256][128]
  __nv_bfloat16 *h, *ht;       // [members * B][ldh], [members * cols][B]
  int ldh;
  const float *t;              // OUT: targets [members * B][24]
  int n_valid;
  double *part;                // OUT: [members][tiles] sums of squared errors
  int *err;
};

// KIND 0: Z = acc + bias, H = silu(Z); 1: the output layer, G = 2 (Y - T) / (24 n)
// and the squared errors; 2: G = acc * silu'(Z)
template <int KIND>
__global__ void __launch_bounds__(TR_NT, 1)
k_train_layer(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
              TrainLayer L) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int s_fail;
  __shared__ double s_red[4];
  const TrainSmem sm = train_smem_of(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = warp & 3, cg = warp >> 2;
  const int member = blockIdx.y, r = blockIdx.x * BM + q * 32 + lane;  // row within the member
  const size_t grow = (size_t) member * L.B + r;
  const unsigned tmem = train_begin(sm, &s_fail);
  const bool ok = train_mma(sm, tmem, &ta, &tb, L.nk, member * L.B + blockIdx.x * BM,
                            member * L.brows, L.bn, L.err, &s_fail);
  const unsigned tl = tmem + ((unsigned) (q * 32) << 16);
  if (ok && KIND != 1) {
    float *zt = L.z + ((size_t) member * (L.B / BM) + blockIdx.x) * (TR_H * BM) + q * 32 + lane;
    const float *bias = KIND == 0 ? L.bias + member * L.pstride : nullptr;
#pragma unroll 1
    for (int c = cg * 64; c < cg * 64 + 64; c += 16) {
      float v[16], zz[16];
      if (KIND == 2) {
#pragma unroll
        for (int i = 0; i < 16; i++) zz[i] = zt[(size_t) (c + i) * BM];
      }
      tmem_ld16(tl + c, v);
      float hv[16];
#pragma unroll
      for (int i = 0; i < 16; i++) {
        if (KIND == 0) {
          const float z = v[i] + __ldg(bias + c + i);
          zt[(size_t) (c + i) * BM] = z;
          hv[i] = z * sigmoidf_(z);
        } else {
          const float z = zz[i], sg = sigmoidf_(z);
          hv[i] = v[i] * sg * (1.f + z * (1.f - sg));
        }
      }
      unsigned w[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const __nv_bfloat162 p2 = __floats2bfloat162_rn(hv[2 * i], hv[2 * i + 1]);
        w[i] = *reinterpret_cast<const unsigned *>(&p2);
        __nv_bfloat16 *ht = L.ht + ((size_t) member * TR_H + c + 2 * i) * L.B + r;
        ht[0] = p2.x;
        ht[L.B] = p2.y;
      }
      uint4 *h = reinterpret_cast<uint4 *>(L.h + grow * L.ldh + c);
      h[0] = make_uint4(w[0], w[1], w[2], w[3]);
      h[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
  }
  if (KIND == 1) {
    double sq = 0.0;
    if (ok && cg == 0) {
      float y[32];
      tmem_ld16(tl, *reinterpret_cast<float(*)[16]>(y));
      tmem_ld16(tl + 16, *reinterpret_cast<float(*)[16]>(y + 16));
      const float *bias = L.bias + member * L.pstride, *t = L.t + grow * TR_OUT;
#pragma unroll
      for (int c = 0; c < TR_OUT; c += 2) {
        float g[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          g[i] = 0.f;
          if (r < L.n_valid) {
            const float d = y[c + i] + __ldg(bias + c + i) - t[c + i];
            sq += (double) d * d;
            g[i] = 2.f * d / ((float) L.n_valid * TR_OUT);
          }
        }
        const __nv_bfloat162 p2 = __floats2bfloat162_rn(g[0], g[1]);
        *reinterpret_cast<__nv_bfloat162 *>(L.h + grow * L.ldh + c) = p2;
        __nv_bfloat16 *ht = L.ht + ((size_t) member * TR_OUT + c) * L.B + r;
        ht[0] = p2.x;
        ht[L.B] = p2.y;
      }
    }
    if (cg == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
      if (lane == 0) s_red[q] = sq;
    }
    __syncthreads();
    if (threadIdx.x == 0)
      L.part[member * gridDim.x + blockIdx.x] = (s_red[0] + s_red[1]) + (s_red[2] + s_red[3]);
  }
  train_end(tmem);
}

// weight gradients dW_l = G_l^T H_{l-1} of layers 0..3, both operands transposed
// (K = the batch, in one accumulator): 128 x 128 tiles, 12 per member
struct TrainDwMaps {
  CUtensorMap a[4], b[4];
};
struct TrainDw {
  int B;
  float *g;
  long nparam, off[4];
  int *err;
};
constexpr int TR_DW_TILES = 12;

__global__ void __launch_bounds__(TR_NT, 1)
k_train_dw(const __grid_constant__ TrainDwMaps maps, TrainDw d) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int s_fail;
  const TrainSmem sm = train_smem_of(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = warp & 3, cg = warp >> 2;
  const int member = blockIdx.y, b = blockIdx.x;
  // layers 1, 2 (256 x 256: 4 tiles each), 0 (256 x 64: 2), 3 (24 x 256: 2)
  const int l = b < 4 ? 1 : b < 8 ? 2 : b < 10 ? 0 : 3;
  const int rt = b < 8 ? (b & 2) >> 1 : b < 10 ? b - 8 : 0;   // row tile
  const int ct = b < 8 ? b & 1 : b < 10 ? 0 : b - 10;         // column tile
  const int arows = l == 3 ? TR_OUT : TR_H, brows = l == 0 ? TR_IN : TR_H, ldw = l == 0 ? 32 : TR_H;
  const int bn = l == 0 ? TR_IN : 128;
  const unsigned tmem = train_begin(sm, &s_fail);
  const bool ok = train_mma(sm, tmem, &maps.a[l], &maps.b[l], d.B / BK, member * arows + rt * BM,
                            member * brows + ct * 128, bn, d.err, &s_fail);
  const int row = rt * BM + q * 32 + lane;
  if (ok) {
    const unsigned tl = tmem + ((unsigned) (q * 32) << 16);
    float *out = d.g + (size_t) member * d.nparam + d.off[l] + (size_t) row * ldw + ct * 128;
#pragma unroll 1
    for (int c = cg * 32; c < min(cg * 32 + 32, min(ldw, 128)); c += 16) {
      float v[16];
      tmem_ld16(tl + c, v);
      if (row < arows)
#pragma unroll
        for (int i = 0; i < 4; i++)
          reinterpret_cast<float4 *>(out + c)[i] =
              make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
  }
  train_end(tmem);
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    check(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q),
          "cuTensorMapEncodeTiled entry point");
    if (!p || q != cudaDriverEntryPointSuccess)
      throw CudaError{cudaErrorNotSupported, "cuTensorMapEncodeTiled unavailable"};
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// 2-D bf16 map over rows x cols (cols contiguous, ld elements per row), box 64 x box_rows
CUtensorMap make_map(const void *ptr, int rows, int cols, int ld, int box_rows) {
  CUtensorMap m;
  cuuint64_t dims[2] = {(cuuint64_t) cols, (cuuint64_t) rows};
  cuuint64_t strides[1] = {(cuuint64_t) ld * 2};
  cuuint32_t box[2] = {(cuuint32_t) BK, (cuuint32_t) box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims,
                           strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw CudaError{cudaErrorInvalidValue, "cuTensorMapEncodeTiled"};
  return m;
}

// Raises a kernel's limit of dynamic shared memory on the current device.  The limit belongs
// to the device, so nothing remembers it for the process: a net sets its kernels' when it is
// made, k_gemm_tn its own at each launch.  Always the same size for a kernel, so that another
// thread's launch finds it large enough.
void allow_smem(const void *kernel, size_t smem) {
  check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem),
        "shared memory limit");
}

template <int BN, int STAGES>
size_t smem_bytes() {
  return 1024 + (size_t) STAGES * (BM * BK * 2 + BN * BK * 2) + (2 * STAGES + 1) * 8 + 16;
}

template <int BN, int STAGES>
void launch(const CUtensorMap &ta, const CUtensorMap &tb, int M, int N, int K, const Epi &ep,
            int *err, cudaStream_t s) {
  const size_t smem = smem_bytes<BN, STAGES>();
  allow_smem((const void *) k_gemm_tn<BN, STAGES>, smem);
  dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN);
  k_gemm_tn<BN, STAGES><<<grid, NT, smem, s>>>(ta, tb, M, N, K, ep, err);
  check(cudaGetLastError(), "k_gemm_tn");
}

}  // namespace

// C = A * B^T with A [M x K] (lda), B [N x K] (ldb), bf16, K % 64 == 0,
// lda, ldb multiples of 8, 16-byte aligned bases.  BN = 32, 64, 128 or 256
// by N (N > 256 is split over grid.y).
void gemm_tn(const void *A, int lda, const void *B, int ldb, int M, int N, int K, float *c, int ldc,
             int *err, cudaStream_t s) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0 || K % BK || lda % 8 || ldb % 8 || (reinterpret_cast<uintptr_t>(A) & 15) ||
      (reinterpret_cast<uintptr_t>(B) & 15))
    throw CudaError{cudaErrorInvalidValue,
                    "gemm_tn: K must be a multiple of 64, leading dimensions multiples of 8"};
  Epi ep{c, ldc};
  const int bn = N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256;
  CUtensorMap ta = make_map(A, M, K, lda, BM);
  CUtensorMap tb = make_map(B, N, K, ldb, bn);
  switch (bn) {
    case 32: launch<32, 4>(ta, tb, M, N, K, ep, err, s); break;
    case 64: launch<64, 4>(ta, tb, M, N, K, ep, err, s); break;
    case 128: launch<128, 4>(ta, tb, M, N, K, ep, err, s); break;
    default: launch<256, 3>(ta, tb, M, N, K, ep, err, s); break;
  }
}

// The tensor maps of a training call (the buffers stay where they are).
struct TrainPlan {
  TrainArgs t;
  CUtensorMap act[7], wts[7];  // forward layers 0..3, backward layers 2, 1, 0
  TrainDwMaps dw;
};

TrainPlan *train_plan(const TrainArgs &t) {
  const int M = t.members, B = t.B;
  auto act = [&](const void *p, int cols) { return make_map(p, M * B, cols, cols, BM); };
  TrainPlan *pl = new TrainPlan;
  try {
    pl->t = t;
    for (int l = 0; l < 4; l++) {
      const int kc = l == 0 ? TR_IN : TR_H, rows = l == 3 ? TR_OUT : TR_H;
      pl->act[l] = act(t.h[l], kc);
      pl->wts[l] = make_map(t.w[l], M * rows, kc, kc, l == 3 ? 32 : TR_H);
      pl->dw.a[l] = make_map(t.gt[l], M * rows, B, B, BM);
      pl->dw.b[l] = make_map(t.ht[l], M * kc, B, B, l == 0 ? TR_IN : 128);
    }
    for (int l = 2; l >= 0; l--) {
      const int kc = l == 2 ? TR_OUTP : TR_H;
      pl->act[6 - l] = act(t.g[l + 1], kc);
      pl->wts[6 - l] = make_map(t.wt[l + 1], M * TR_H, kc, kc, TR_H);
    }
  } catch (...) {
    delete pl;
    throw;
  }
  return pl;
}

void train_plan_free(TrainPlan *p) { delete p; }

// One step's forward and backward passes and weight gradients; the squared
// errors go to `loss` ([members][B / 128])
void train_passes(const TrainPlan &pl, double *loss, cudaStream_t s) {
  const TrainArgs &t = pl.t;
  const size_t smem = train_smem();
  auto bf = [](void *p) { return static_cast<__nv_bfloat16 *>(p); };
  const dim3 grid(t.B / BM, t.members);
  TrainLayer L{};
  L.B = t.B;
  L.pstride = t.pstride;
  L.n_valid = t.n_valid;
  L.t = t.tb;
  L.part = loss;
  L.err = t.err;
  // forward: h_l = silu(h_{l-1} W_l^T + b_l), then the output layer
  for (int l = 0; l < 3; l++) {
    L.nk = l == 0 ? 1 : TR_H / BK;
    L.bn = L.brows = L.ldh = TR_H;
    L.bias = t.p + t.ob[l];
    L.z = t.z[l];
    L.h = bf(t.h[l + 1]);
    L.ht = bf(t.ht[l + 1]);
    k_train_layer<0><<<grid, TR_NT, smem, s>>>(pl.act[l], pl.wts[l], L);
  }
  L.nk = TR_H / BK;
  L.bn = 32;
  L.brows = TR_OUT;
  L.bias = t.p + t.ob[3];
  L.h = bf(t.g[3]);
  L.ldh = TR_OUTP;
  L.ht = bf(t.gt[3]);
  k_train_layer<1><<<grid, TR_NT, smem, s>>>(pl.act[3], pl.wts[3], L);
  // backward: g_l = (g_{l+1} W_{l+1}) silu'(z_l)
  for (int l = 2; l >= 0; l--) {
    L.nk = (l == 2 ? TR_OUTP : TR_H) / BK;
    L.bn = L.brows = L.ldh = TR_H;
    L.z = t.z[l];
    L.h = bf(t.g[l]);
    L.ht = bf(t.gt[l]);
    k_train_layer<2><<<grid, TR_NT, smem, s>>>(pl.act[6 - l], pl.wts[6 - l], L);
  }
  TrainDw d{};
  d.B = t.B;
  d.g = t.grad;
  d.nparam = t.pstride;
  d.err = t.err;
  for (int l = 0; l < 4; l++) d.off[l] = t.ow[l];
  k_train_dw<<<dim3(TR_DW_TILES, t.members), TR_NT, smem, s>>>(pl.dw, d);
  check(cudaGetLastError(), "train_passes");
}

static size_t ensemble_smem(int members) {
  return 1024 + ENS_X_BYTES + ENS_A_BYTES + (size_t) ENS_STAGES * ENS_W_BYTES +
         sizeof(float) * members * ENS_BSTRIDE + (2 * ENS_STAGES + 2) * 8 + 16;
}

void allow_net() {
  for (const void *k : {(const void *) k_train_layer<0>, (const void *) k_train_layer<1>,
                        (const void *) k_train_layer<2>, (const void *) k_train_dw})
    allow_smem(k, train_smem());
  allow_smem((const void *) k_mlp_ensemble, ensemble_smem(ENS_MAX_MEMBERS));
}

// The fused ensemble on normalised bf16 features xf[n][64]; weights stacked
// over the members: w1s[m*256][64], w2s/w3s[m*256][256], w4s[m*24][256];
// bias[m][792] (b1, b2, b3, b4).
void mlp_ensemble(const void *xf, int n, const void *w1s, const void *w2s, const void *w3s,
                  const void *w4s, const float *bias, int members, const float *norm, float *mean,
                  float *spread, int *err, cudaStream_t s, const int *count) {
  if (n <= 0) return;
  if (members < 1 || members > ENS_MAX_MEMBERS)
    throw CudaError{cudaErrorInvalidValue, "mlp_ensemble: 1..4 members"};
  CUtensorMap tx = make_map(xf, n, 64, 64, BM);
  CUtensorMap t1 = make_map(w1s, members * ENS_H, 64, 64, ENS_H);
  CUtensorMap t2 = make_map(w2s, members * ENS_H, ENS_H, ENS_H, ENS_H);
  CUtensorMap t3 = make_map(w3s, members * ENS_H, ENS_H, ENS_H, ENS_H);
  CUtensorMap t4 = make_map(w4s, members * ENS_OUT, ENS_H, ENS_H, 32);
  const size_t smem = ensemble_smem(members);
  EnsArgs a{bias, norm, mean, spread, n, members, err, count};
  k_mlp_ensemble<<<(n + BM - 1) / BM, ENS_NT, smem, s>>>(tx, t1, t2, t3, t4, a);
  check(cudaGetLastError(), "k_mlp_ensemble");
}

}  // namespace gemm
}  // namespace cacg
