// The nodal-force surrogate: an ensemble of MLPs 32 -> 256 -> 256 -> 256 -> 24
// (SiLU) that maps an element's 24 nodal displacements (about their mean,
// relative to the ideal lattice) and 8 nodal densities to its 24 nodal forces.
//
// Every matrix product, forward and backward, runs on the tensor cores (BF16
// operands, FP32 accumulation, k_gemm.cu), all members of a step together.  Master weights,
// Adam moments and gradients are FP32; activations cross layers as BF16 and
// pre-activations are kept in FP32 for the SiLU derivative.  The reference has
// no counterpart: it evaluates every element by integration-point quadrature.
//
// Parameters per member, flattened: W1[256][32] b1[256] W2[256][256] b2
// W3[256][256] b3 W4[24][256] b4[24]; the step's arrays are gemm::TrainArgs.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "cacg.h"
#include "internal.h"

namespace cacg {
namespace mlp {

using bf16 = __nv_bfloat16;

namespace {

constexpr int NIN = MLP_IN, NINP = 64, NH = MLP_HIDDEN, NOUT = MLP_OUT, NGP = 64;
static_assert(NH % 64 == 0 && NIN <= NINP && NOUT <= NGP, "layer shapes the GEMM tiles support");
constexpr long oW1 = 0, ob1 = oW1 + (long) NH * NIN, oW2 = ob1 + NH, ob2 = oW2 + (long) NH * NH,
               oW3 = ob2 + NH, ob3 = oW3 + (long) NH * NH, oW4 = ob3 + NH,
               ob4 = oW4 + (long) NOUT * NH, NPARAM = ob4 + NOUT;

inline int nblk(long long n, int t) { return (int) ((n + t - 1) / t); }

// The current parameters' BF16 copies, stacked over the members: forward
// weights w[0..3] ([256][64] K padded, [256][256] twice, [24][256]), transposed
// wt[1..3] ([256][256] twice, [256][64] padded), biases for inference [792].
struct Copies {
  bf16 *w[4], *wt[4];
  float *bias;
};

constexpr int BIASES = 3 * NH + NOUT;
constexpr long WEIGHTS = NPARAM - BIASES;

// writes parameter i of a member to its copies
__device__ __forceinline__ void put_copy(const Copies &c, int member, int layer, int r, int col,
                                         float v) {
  const bf16 b = __float2bfloat16(v);
  if (layer == 0) {
    c.w[0][((size_t) member * NH + r) * NINP + col] = b;
  } else if (layer < 3) {
    c.w[layer][((size_t) member * NH + r) * NH + col] = b;
    c.wt[layer][((size_t) member * NH + col) * NH + r] = b;
  } else {
    c.w[3][((size_t) member * NOUT + r) * NH + col] = b;
    c.wt[3][((size_t) member * NH + col) * NGP + r] = b;
  }
}

enum { UPDATE_COPY = 0, UPDATE_GRAD = 1, UPDATE_ADAM = 2 };

struct UpdateArgs {
  float *p, *m, *v, *g;   // [members][NPARAM]; g holds the weight gradients
  const bf16 *gt[4];      // gradients at the layers' outputs, transposed [members * rows][B]
  int B, first;           // first: member of blockIdx.y == 0
  float lr, b1, b2, eps, bc1, bc2;
  Copies c;
};

// blockIdx.y: member; the first WB blocks take the weights (a thread each), the
// others the biases (a warp each: the column sum of the gradient, by 256 rows,
// of these by eights, in order: the same bits on every run, where atomics add the
// parts as blocks arrive)
constexpr int UB = 256;
constexpr int WB = (int) ((WEIGHTS + UB - 1) / UB), BB = (BIASES + UB / 32 - 1) / (UB / 32);

template <int MODE>
__global__ void __launch_bounds__(UB) k_update(UpdateArgs a) {
  const int member = a.first + blockIdx.y;
  long off;            // in the member's parameters
  int layer, r, col;   // weight (r, col), or bias r with col < 0
  float g = 0.f;
  if ((int) blockIdx.x < WB) {
    long i = blockIdx.x * (long) UB + threadIdx.x;
    if (i >= WEIGHTS) return;
    layer = 0;
    int cols = NIN;
    if (i >= (long) NH * NIN) {
      i -= (long) NH * NIN;
      layer = i < (long) NH * NH ? 1 : i < 2L * NH * NH ? 2 : 3;
      i -= (long) (layer - 1) * NH * NH;
      cols = NH;
    }
    r = (int) (i / cols);
    col = (int) (i % cols);
    off = (layer == 0 ? oW1 : layer == 1 ? oW2 : layer == 2 ? oW3 : oW4) + i;
    if (MODE != UPDATE_COPY) g = a.g[(size_t) member * NPARAM + off];
  } else {
    const int j = ((int) blockIdx.x - WB) * (UB / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= BIASES) return;
    layer = j / NH;
    r = j % NH;
    col = -1;
    off = (layer == 0 ? ob1 : layer == 1 ? ob2 : layer == 2 ? ob3 : ob4) + r;
    if (MODE != UPDATE_COPY) {
      const int rows = layer == 3 ? NOUT : NH;
      const bf16 *q = a.gt[layer] + ((size_t) blockIdx.y * rows + r) * a.B;
      // four groups of 256 rows at a time, a lane per group and row modulo 8
      for (int r0 = 0; r0 < a.B; r0 += 1024) {
        const int first = r0 + (lane >> 3) * 256;
        float t = 0.f, s = 0.f;
        for (int k = first + (lane & 7); k < min(first + 256, a.B); k += 8)
          s += __bfloat162float(q[k]);
        for (int w = 0; w < 4; w++) {
          t = 0.f;
          for (int y = 0; y < 8; y++) t += __shfl_sync(0xffffffffu, s, 8 * w + y);
          if (r0 + 256 * w < a.B) g += t;
        }
      }
    }
    if (lane != 0) return;
  }
  const size_t at = (size_t) member * NPARAM + off;
  if (MODE == UPDATE_GRAD) {
    a.g[at] = g;
    return;
  }
  float p = a.p[at];
  if (MODE == UPDATE_ADAM) {
    const float mi = __fmaf_rn(1.f - a.b1, g, __fmul_rn(a.b1, a.m[at]));
    const float vi = __fmaf_rn(__fmul_rn(1.f - a.b2, g), g, __fmul_rn(a.b2, a.v[at]));
    a.m[at] = mi;
    a.v[at] = vi;
    p -= a.lr * (mi / a.bc1) / (sqrtf(vi / a.bc2) + a.eps);
    a.p[at] = p;
  }
  if (col >= 0) put_copy(a.c, member, layer, r, col, p);
  else a.c.bias[(size_t) member * BIASES + layer * NH + r] = p;
}

// Column means and standard deviations of two [n][cols] arrays, a block each: FP32
// sums down the rows in order, as an array library forms them (so that a data set is
// normalised to the same bits), the quotients by n in FP64 where wide is set.  Bound by
// the chain of additions, 4 cycles a row: the rows come through shared memory, MO_STAGES
// chunks ahead.  65,536 rows of 32 and 24: 1.2 ms with the copies, by the host 7.3.
constexpr int MO_NT = 256, MO_ROWS = 64, MO_STAGES = 4;
struct Moments {
  const float *a[2];
  int cols[2];
  float *mean[2], *std[2];
};

__global__ void __launch_bounds__(MO_NT) k_moments(Moments q, long n, int wide) {
  __shared__ __align__(16) float s_buf[MO_STAGES][MO_ROWS * NIN];
  const int cols = q.cols[blockIdx.x], tid = threadIdx.x;
  const float *a = q.a[blockIdx.x];
  const long total = n * cols, chunk = (long) MO_ROWS * cols, chunks = (n + MO_ROWS - 1) / MO_ROWS;
  auto fetch = [&](long c) {
    if (c < chunks) {
      const float *src = a + c * chunk;
      const long len = min(chunk, total - c * chunk);  // a multiple of 4 floats
      const unsigned dst = (unsigned) __cvta_generic_to_shared(s_buf[c % MO_STAGES]);
      for (int i = 4 * tid; i < len; i += 4 * MO_NT)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 4 * i), "l"(src + i));
    }
    asm volatile("cp.async.commit_group;");
  };
  auto quotient = [&](float v) {
    return wide ? (float) ((double) v / (double) n) : __fdiv_rn(v, (float) n);
  };
  float mean = 0.f;
  for (int pass = 0; pass < 2; pass++) {
    float s = 0.f;
    for (int c = 0; c < MO_STAGES - 1; c++) fetch(c);
    for (long c = 0; c < chunks; c++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(MO_STAGES - 2));
      __syncthreads();
      fetch(c + MO_STAGES - 1);
      if (tid < cols) {
        const float *b = s_buf[c % MO_STAGES] + tid;
        const int rows = (int) min((long) MO_ROWS, n - c * MO_ROWS);
        auto take = [&](float v) {
          if (pass) {
            v = __fsub_rn(v, mean);
            v = __fmul_rn(v, v);
          }
          s = __fadd_rn(s, v);
        };
        if (rows == MO_ROWS) {
#pragma unroll 16
          for (int r = 0; r < MO_ROWS; r++) take(b[r * cols]);
        } else {
          for (int r = 0; r < rows; r++) take(b[r * cols]);
        }
      }
    }
    __syncthreads();
    if (pass == 0) mean = quotient(s);
    else if (tid < cols) {
      q.mean[blockIdx.x][tid] = mean;
      q.std[blockIdx.x][tid] = __fsqrt_rn(quotient(s));
    }
  }
}

// sums of the squares of the rows' 24 values in FP64, by eight strands added in pairs
__global__ void k_row_squares(const float *__restrict__ t, long n, double *__restrict__ out) {
  const long i = blockIdx.x * (long) blockDim.x + threadIdx.x;
  if (i >= n) return;
  double r[8];
#pragma unroll
  for (int k = 0; k < NOUT; k++) {
    const double v = t[i * NOUT + k], w = __dmul_rn(v, v);
    r[k % 8] = k < 8 ? w : __dadd_rn(r[k % 8], w);
  }
  out[i] = __dadd_rn(__dadd_rn(__dadd_rn(r[0], r[1]), __dadd_rn(r[2], r[3])),
                     __dadd_rn(__dadd_rn(r[4], r[5]), __dadd_rn(r[6], r[7])));
}

// normalised features as bf16 [n][64]: (x - mean) * inv_std, zero padded
__global__ void k_features(const float *__restrict__ x, long n, const float *__restrict__ norm,
                           bf16 *__restrict__ out) {
  long i = blockIdx.x * (long) blockDim.x + threadIdx.x;
  if (i >= n * NINP) return;
  long r = i / NINP;
  int c = (int) (i % NINP);
  float v = 0.f;
  if (c < NIN) v = (x[r * NIN + c] - norm[c]) * norm[NIN + c];
  out[i] = __float2bfloat16(v);
}

// normalised targets: (t - out_mean) / out_std
__global__ void k_targets(const float *__restrict__ t, long n, const float *__restrict__ norm,
                          float *__restrict__ out) {
  long i = blockIdx.x * (long) blockDim.x + threadIdx.x;
  if (i >= n * NOUT) return;
  int c = (int) (i % NOUT);
  out[i] = (t[i] - norm[2 * NIN + c]) / norm[2 * NIN + NOUT + c];
}

// The members' batches: features x0 [members * B][64] and their transpose
// [members * 64][B], targets tb [members * B][24]; row r of member m is sample
// idx[m * istride + r] (idx null: r), zero for r >= n
__global__ void __launch_bounds__(256)
k_gather(const bf16 *__restrict__ xall, const float *__restrict__ tall, const int *__restrict__ idx,
         long istride, int n, int B, bf16 *__restrict__ x0, bf16 *__restrict__ x0t,
         float *__restrict__ tb) {
  __shared__ bf16 t[32][NINP + 2];
  const int member = blockIdx.y, r0 = blockIdx.x * 32;
  for (int k = threadIdx.x; k < 32 * NINP; k += 256) {
    const int r = k / NINP, c = k % NINP;
    const int src = r0 + r >= n ? -1 : idx ? idx[member * istride + r0 + r] : r0 + r;
    const bf16 v = src >= 0 ? xall[(long) src * NINP + c] : __float2bfloat16(0.f);
    const size_t row = (size_t) member * B + r0 + r;
    x0[row * NINP + c] = v;
    t[r][c] = v;
    if (c < NOUT) tb[row * NOUT + c] = src >= 0 ? tall[(long) src * NOUT + c] : 0.f;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 32 * NINP; k += 256) {
    const int c = k / 32, r = k % 32;
    x0t[((size_t) member * NINP + c) * B + r0 + r] = t[r][c];
  }
}

// splitmix64: seeded, platform-independent initialisation
struct Rng {
  unsigned long long s;
  unsigned long long next() {
    unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
  void skip(unsigned long long n) { s += n * 0x9E3779B97F4A7C15ull; }
  double uniform() { return (next() >> 11) * (1.0 / 9007199254740992.0); }
};

}  // namespace

struct Net {
  int device = 0, members = 0;
  cudaStream_t stream = nullptr;
  float norm[2 * NIN + 2 * NOUT];  // in_mean, in_inv_std, out_mean, out_std
  double force_scale = 1.0;        // rms nodal-force magnitude of the training targets
  long long adam_steps = 0;
  std::string err;
  DBuf<float> d_norm;
  // per member, stacked: parameters, Adam moments, gradients, BF16 copies
  DBuf<float> p, m, v, g, bias;
  DBuf<bf16> w[4], wt[4];
  // one step's arrays (see gemm::TrainArgs)
  DBuf<bf16> h[4], ht[4], gr[4], grt[4];
  DBuf<float> z[3], tb;
  DBuf<double> loss;
  DBuf<int> errflag;
  size_t g4_rows = 0;  // rows of gr[3] whose padding is zero
  // a call's data set and results: kept for the next call (cudaMalloc and
  // cudaFree of a prediction's buffers cost more than its kernel), unless larger
  // than KEEP_BYTES
  DBuf<float> raw, rt, tf, dm, ds;
  DBuf<bf16> xf;
  static constexpr size_t KEEP_BYTES = 64u << 20;
  void trim() {
    for (DBuf<float> *b : {&raw, &rt, &tf, &dm, &ds})
      if (b->cap * sizeof(float) > KEEP_BYTES) b->release();
    if (xf.cap * sizeof(bf16) > KEEP_BYTES) xf.release();
  }

  void sync() { check(cudaStreamSynchronize(stream), "mlp sync"); }

  void ensure_err(cudaStream_t s) {
    if (errflag.p) return;
    errflag.ensure(1, s);
    check(cudaMemsetAsync(errflag.p, 0, sizeof(int), s), "errflag");
  }

  void upload_norm() {
    d_norm.ensure(2 * NIN + 2 * NOUT, stream);
    check(cudaMemcpyAsync(d_norm.p, norm, sizeof(norm), cudaMemcpyHostToDevice, stream), "norm");
  }

  void init_params(unsigned long long seed) {
    Rng rng{seed};
    std::vector<float> hp((size_t) members * NPARAM, 0.f);
    for (int k = 0; k < members; k++) {
      float *q = hp.data() + (size_t) k * NPARAM;
      auto fill = [&](long off, int rows, int cols, double gain) {
        double a = gain * std::sqrt(3.0 / cols);
        for (long i = 0; i < (long) rows * cols; i++) q[off + i] = (float) ((2 * rng.uniform() - 1) * a);
      };
      fill(oW1, NH, NIN, 1.0);
      fill(oW2, NH, NH, 1.0);
      fill(oW3, NH, NH, 1.0);
      fill(oW4, NOUT, NH, 0.1);
    }
    const size_t np = hp.size(), mm = (size_t) members;
    for (DBuf<float> *b : {&p, &m, &v, &g}) b->ensure(np, stream);
    bias.ensure(mm * BIASES, stream);
    w[0].ensure(mm * NH * NINP, stream);
    w[1].ensure(mm * NH * NH, stream);
    w[2].ensure(mm * NH * NH, stream);
    w[3].ensure(mm * NOUT * NH, stream);
    wt[1].ensure(mm * NH * NH, stream);
    wt[2].ensure(mm * NH * NH, stream);
    wt[3].ensure(mm * NH * NGP, stream);
    // the padding of W1 and W4^T stays zero
    check(cudaMemsetAsync(w[0].p, 0, sizeof(bf16) * mm * NH * NINP, stream), "w1");
    check(cudaMemsetAsync(wt[3].p, 0, sizeof(bf16) * mm * NH * NGP, stream), "w4t");
    check(cudaMemcpyAsync(p.p, hp.data(), sizeof(float) * np, cudaMemcpyHostToDevice, stream), "params");
    check(cudaMemsetAsync(m.p, 0, sizeof(float) * np, stream), "adam m");
    check(cudaMemsetAsync(v.p, 0, sizeof(float) * np, stream), "adam v");
    refresh(0, members);
    sync();
  }

  UpdateArgs update_args(int first) {
    UpdateArgs a{};
    a.p = p.p;
    a.m = m.p;
    a.v = v.p;
    a.g = g.p;
    a.first = first;
    for (int l = 0; l < 4; l++) {
      a.c.w[l] = w[l].p;
      a.c.wt[l] = wt[l].p;
      a.gt[l] = grt[l].p;
    }
    a.c.bias = bias.p;
    return a;
  }

  // BF16 copies of the members' weights (forward and transposed)
  void refresh(int first, int count) {
    k_update<UPDATE_COPY><<<dim3(WB + BB, count), UB, 0, stream>>>(update_args(first));
    check(cudaGetLastError(), "mlp refresh");
  }

  // `count` members from `first` with B rows each
  gemm::TrainArgs batch(int first, int count, int B, int n_valid) {
    cudaStream_t s = stream;
    const size_t b = (size_t) count * B;
    h[0].ensure(b * NINP, s);
    ht[0].ensure(b * NINP, s);
    for (int l = 1; l < 4; l++) {
      h[l].ensure(b * NH, s);
      ht[l].ensure(b * NH, s);
      gr[l - 1].ensure(b * NH, s);
      grt[l - 1].ensure(b * NH, s);
      z[l - 1].ensure(b * NH, s);
    }
    if (gr[3].cap < b * NGP) g4_rows = 0;
    gr[3].ensure(b * NGP, s);
    if (g4_rows < b) {  // columns 24..63 stay zero
      check(cudaMemsetAsync(gr[3].p, 0, sizeof(bf16) * b * NGP, s), "g4");
      g4_rows = b;
    }
    grt[3].ensure(b * NOUT, s);
    tb.ensure(b * NOUT, s);
    ensure_err(s);
    gemm::TrainArgs t{};
    t.members = count;
    t.B = B;
    t.n_valid = n_valid;
    t.p = p.p + (size_t) first * NPARAM;
    t.pstride = NPARAM;
    const long ow[4] = {oW1, oW2, oW3, oW4}, ob[4] = {ob1, ob2, ob3, ob4};
    const size_t wrow[4] = {NH * NINP, NH * NH, NH * NH, NOUT * NH},
                 wtrow[4] = {0, NH * NH, NH * NH, NH * NGP};
    for (int l = 0; l < 4; l++) {
      t.ow[l] = ow[l];
      t.ob[l] = ob[l];
      t.h[l] = h[l].p;
      t.ht[l] = ht[l].p;
      t.g[l] = gr[l].p;
      t.gt[l] = grt[l].p;
      t.w[l] = w[l].p + first * wrow[l];
      t.wt[l] = l ? wt[l].p + first * wtrow[l] : nullptr;
      if (l < 3) t.z[l] = z[l].p;
    }
    t.tb = tb.p;
    t.grad = g.p + (size_t) first * NPARAM;
    t.err = errflag.p;
    return t;
  }

  // the step's arrays given back
  void release_batch() {
    for (int l = 0; l < 4; l++)
      for (auto *b : {&h[l], &ht[l], &gr[l], &grt[l]}) b->release();
    for (auto &b : z) b.release();
    tb.release();
    g4_rows = 0;
  }

  void gather(const gemm::TrainArgs &t, const bf16 *xall, const float *tall, const int *idx,
              long istride, int n) {
    k_gather<<<dim3(t.B / 32, t.members), 256, 0, stream>>>(xall, tall, idx, istride, n, t.B, h[0].p,
                                                           ht[0].p, tb.p);
    check(cudaGetLastError(), "gather");
  }

  void check_err() {
    int f = 0;
    check(cudaMemcpyAsync(&f, errflag.p, sizeof(int), cudaMemcpyDeviceToHost, stream), "errflag");
    sync();
    if (f) throw CudaError{cudaErrorLaunchTimeout, "tensor-core GEMM: a bounded wait ran out"};
  }

  // means and deviations of a data set (in, then out), sums of its targets' squares
  void moments(const float *x, const float *t, long long n, int wide, float *const out[4],
               double *row_squares) {
    cudaStream_t s = stream;
    constexpr int C = NIN + NOUT;
    raw.ensure((size_t) n * NIN, s);
    rt.ensure((size_t) n * NOUT, s);
    tf.ensure((size_t) n * 2, s);
    dm.ensure(2 * C, s);
    double *rows = reinterpret_cast<double *>(tf.p);
    check(cudaMemcpyAsync(raw.p, x, sizeof(float) * n * NIN, cudaMemcpyHostToDevice, s), "x");
    check(cudaMemcpyAsync(rt.p, t, sizeof(float) * n * NOUT, cudaMemcpyHostToDevice, s), "t");
    const Moments q{{raw.p, rt.p}, {NIN, NOUT}, {dm.p, dm.p + 2 * NIN}, {dm.p + NIN, dm.p + 2 * NIN + NOUT}};
    k_moments<<<2, MO_NT, 0, s>>>(q, (long) n, wide);
    k_row_squares<<<nblk(n, 256), 256, 0, s>>>(rt.p, (long) n, rows);
    check(cudaGetLastError(), "moments");
    float h[2 * C];
    check(cudaMemcpyAsync(h, dm.p, sizeof h, cudaMemcpyDeviceToHost, s), "moments");
    check(cudaMemcpyAsync(row_squares, rows, sizeof(double) * n, cudaMemcpyDeviceToHost, s), "rows");
    sync();
    const int off[4] = {0, NIN, 2 * NIN, 2 * NIN + NOUT}, len[4] = {NIN, NIN, NOUT, NOUT};
    for (int k = 0; k < 4; k++) std::memcpy(out[k], h + off[k], sizeof(float) * len[k]);
    trim();
  }

  // the members' gradients into g
  void gradients(const gemm::TrainArgs &t, int first) {
    UpdateArgs a = update_args(first);
    a.B = t.B;
    k_update<UPDATE_GRAD><<<dim3(WB + BB, t.members), UB, 0, stream>>>(a);
    check(cudaGetLastError(), "gradients");
  }

  // of t's members, the first of which is `first`
  void adam(const gemm::TrainArgs &t, int first, float lr) {
    UpdateArgs a = update_args(first);
    a.B = t.B;
    a.lr = lr;
    a.b1 = 0.9f;
    a.b2 = 0.999f;
    a.eps = 1e-8f;
    const double step = (double) adam_steps + 1;
    a.bc1 = (float) (1 - std::pow(a.b1, step));
    a.bc2 = (float) (1 - std::pow(a.b2, step));
    k_update<UPDATE_ADAM><<<dim3(WB + BB, t.members), UB, 0, stream>>>(a);
    check(cudaGetLastError(), "adam");
  }

  // ensemble prediction on normalised bf16 features already on the device:
  // one fused launch over all members and layers (gemm::mlp_ensemble)
  void predict_device(const bf16 *xf, long long n, float *mean, float *spread, cudaStream_t s,
                      const int *dcount = nullptr) {
    if (n <= 0) return;
    ensure_err(s);
    gemm::mlp_ensemble(xf, (int) n, w[0].p, w[1].p, w[2].p, w[3].p, bias.p, members, d_norm.p, mean,
                       spread, errflag.p, s, dcount);
  }
};

Net *net_of(cacg_mlp_t *m);
const float *norm_device(const Net *n) { return n->d_norm.p; }
double force_scale(const Net *n) { return n->force_scale; }
int members(const Net *n) { return n->members; }
void predict(Net *n, const void *xf, long long count, float *mean, float *spread, cudaStream_t s,
             const int *dcount) {
  n->ensure_err(s);
  n->predict_device(static_cast<const bf16 *>(xf), count, mean, spread, s, dcount);
}
void check_error(Net *n, cudaStream_t s) {
  int v = 0;
  check(cudaMemcpyAsync(&v, n->errflag.p, sizeof(int), cudaMemcpyDeviceToHost, s), "errflag");
  check(cudaStreamSynchronize(s), "errflag sync");
  if (v) throw CudaError{cudaErrorLaunchTimeout, "tensor-core GEMM: a bounded wait ran out"};
}

void features_bf16(const float *x, long long n, const float *norm, bf16 *out, cudaStream_t s) {
  k_features<<<nblk(n * NINP, 256), 256, 0, s>>>(x, n, norm, out);
  check(cudaGetLastError(), "features");
}

void targets(const float *t, long long n, const float *norm, float *out, cudaStream_t s) {
  k_targets<<<nblk(n * NOUT, 256), 256, 0, s>>>(t, n, norm, out);
  check(cudaGetLastError(), "targets");
}

}  // namespace mlp
}  // namespace cacg

// ------------------------------------------------------------------ C ABI

using cacg::CudaError;
using cacg::mlp::Net;
using cacg::mlp::bf16;

struct cacg_mlp_t {
  Net net;
};

namespace cacg {
namespace mlp {
Net *net_of(cacg_mlp_t *m) { return m ? &m->net : nullptr; }
}  // namespace mlp
}  // namespace cacg

namespace {

struct MlpError {
  int code;
  std::string msg;
};

#define MLP_BEGIN             \
  if (!m) return CACG_EINVAL; \
  try {                       \
    cacg::check(cudaSetDevice(m->net.device), "cudaSetDevice");
// (an error leaves nothing of the call in flight: a copy from or to the caller's pinned
// memory may still run)
#define MLP_END                                                            \
  return CACG_OK;                                                          \
  }                                                                        \
  catch (const MlpError &e) {                                              \
    m->net.err = e.msg;                                                    \
    return e.code;                                                         \
  }                                                                        \
  catch (const CudaError &e) {                                             \
    cudaStreamSynchronize(m->net.stream);                                  \
    m->net.err = std::string(e.where) + ": " + cudaGetErrorString(e.code); \
    return CACG_ECUDA;                                                     \
  }                                                                        \
  catch (const std::bad_alloc &) {                                         \
    cudaStreamSynchronize(m->net.stream);                                  \
    m->net.err = "host allocation failed";                                 \
    return CACG_ENOMEM;                                                    \
  }

void need(bool ok, const char *msg) {
  if (!ok) throw MlpError{CACG_EINVAL, msg};
}

using namespace cacg::mlp;

constexpr int MLP_IN = cacg::MLP_IN, MLP_OUT = cacg::MLP_OUT, MLP_HIDDEN = cacg::MLP_HIDDEN;
constexpr long kNParam = (long) MLP_HIDDEN * MLP_IN + MLP_HIDDEN +
                         2L * (MLP_HIDDEN * MLP_HIDDEN + MLP_HIDDEN) + (long) MLP_OUT * MLP_HIDDEN +
                         MLP_OUT;

struct Plan {
  cacg::gemm::TrainPlan *p;
  explicit Plan(const cacg::gemm::TrainArgs &t) : p(cacg::gemm::train_plan(t)) {}
  ~Plan() { cacg::gemm::train_plan_free(p); }
  Plan(const Plan &) = delete;
  Plan &operator=(const Plan &) = delete;
};

// host tasks on threads of their own; a task whose thread cannot be started
// runs at once.  The destructor waits for all of them.
struct Workers {
  std::vector<std::thread> t;
  template <class F>
  void run(F f) {
    try {
      t.reserve(t.size() + 1);
      t.emplace_back(f);
    } catch (const std::exception &) {
      f();
    }
  }
  void wait() {
    for (std::thread &x : t) x.join();
    t.clear();
  }
  ~Workers() { wait(); }
};

// upload normalised features (bf16 [n][64]) and targets (fp32 [n][24]) into the
// net's data buffers
void upload_set(Net &N, const float *x, const float *t, long long n) {
  cudaStream_t s = N.stream;
  N.raw.ensure((size_t) n * MLP_IN + 1, s);
  cacg::check(cudaMemcpyAsync(N.raw.p, x, sizeof(float) * n * MLP_IN, cudaMemcpyHostToDevice, s), "x");
  N.xf.ensure((size_t) n * 64 + 64, s);
  cacg::mlp::features_bf16(N.raw.p, n, N.d_norm.p, N.xf.p, s);
  if (t) {
    N.rt.ensure((size_t) n * MLP_OUT + 1, s);
    cacg::check(cudaMemcpyAsync(N.rt.p, t, sizeof(float) * n * MLP_OUT, cudaMemcpyHostToDevice, s), "t");
    N.tf.ensure((size_t) n * MLP_OUT + 1, s);
    cacg::mlp::targets(N.rt.p, n, N.d_norm.p, N.tf.p, s);
  }
  // large ones make room for what the call needs next
  for (cacg::DBuf<float> *b : {&N.raw, &N.rt})
    if (b->cap * sizeof(float) > Net::KEEP_BYTES) {
      N.sync();
      b->release();
    }
}

}  // namespace

extern "C" {

int cacg_mlp_create(cacg_mlp *out, int device, int members, unsigned long long seed) {
  if (!out || members < 1 || members > 4) return CACG_EINVAL;
  *out = nullptr;
  cacg_mlp m = new (std::nothrow) cacg_mlp_t;
  if (!m) return CACG_ENOMEM;
  m->net.device = device;
  m->net.members = members;
  int rc = CACG_OK;
  try {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n)
      throw MlpError{CACG_ECUDA, "no CUDA device"};
    cacg::check(cudaSetDevice(device), "cudaSetDevice");
    cacg::check(cudaStreamCreateWithFlags(&m->net.stream, cudaStreamNonBlocking), "stream");
    for (int i = 0; i < MLP_IN; i++) m->net.norm[i] = 0.f, m->net.norm[MLP_IN + i] = 1.f;
    for (int i = 0; i < MLP_OUT; i++)
      m->net.norm[2 * MLP_IN + i] = 0.f, m->net.norm[2 * MLP_IN + MLP_OUT + i] = 1.f;
    cacg::gemm::allow_net();
    m->net.upload_norm();
    m->net.init_params(seed);
  } catch (const MlpError &e) {
    rc = e.code;
  } catch (const CudaError &) {
    rc = CACG_ECUDA;
  }
  if (rc != CACG_OK) {
    delete m;
    return rc;
  }
  *out = m;
  return CACG_OK;
}

int cacg_mlp_destroy(cacg_mlp m) {
  if (!m) return CACG_OK;
  cudaSetDevice(m->net.device);
  if (m->net.stream) cudaStreamSynchronize(m->net.stream);
  Net &N = m->net;
  for (auto *b : {&N.p, &N.m, &N.v, &N.g, &N.bias, &N.d_norm, &N.tb, &N.raw, &N.rt, &N.tf, &N.dm, &N.ds}) b->release();
  for (int l = 0; l < 4; l++)
    for (auto *b : {&N.w[l], &N.wt[l], &N.h[l], &N.ht[l], &N.gr[l], &N.grt[l]}) b->release();
  for (auto &b : N.z) b.release();
  N.loss.release();
  N.xf.release();
  N.errflag.release();
  if (N.stream) cudaStreamDestroy(N.stream);
  delete m;
  return CACG_OK;
}

const char *cacg_mlp_error(cacg_mlp m) { return m ? m->net.err.c_str() : "null handle"; }

int cacg_mlp_sizes(cacg_mlp m, long long *sizes, int n) {
  MLP_BEGIN
  need(sizes && n > 0, "bad output array");
  long long v[6] = {m->net.members, kNParam, MLP_IN, MLP_OUT, MLP_HIDDEN, m->net.adam_steps};
  for (int i = 0; i < n && i < 6; i++) sizes[i] = v[i];
  MLP_END
}

int cacg_mlp_get_params(cacg_mlp m, int member, float *p) {
  MLP_BEGIN
  need(p && member >= 0 && member < m->net.members, "bad member or array");
  cacg::check(cudaMemcpyAsync(p, m->net.p.p + (size_t) member * kNParam, sizeof(float) * kNParam,
                              cudaMemcpyDeviceToHost, m->net.stream), "params");
  m->net.sync();
  MLP_END
}

int cacg_mlp_set_params(cacg_mlp m, int member, const float *p) {
  MLP_BEGIN
  need(p && member >= 0 && member < m->net.members, "bad member or array");
  cacg::check(cudaMemcpyAsync(m->net.p.p + (size_t) member * kNParam, p, sizeof(float) * kNParam,
                              cudaMemcpyHostToDevice, m->net.stream), "params");
  m->net.refresh(member, 1);
  m->net.sync();
  MLP_END
}

int cacg_mlp_moments(cacg_mlp m, const float *x, const float *t, long long n, int wide, float *in_mean,
                     float *in_std, float *out_mean, float *out_std, double *row_squares) {
  MLP_BEGIN
  need(x && t && in_mean && in_std && out_mean && out_std && row_squares && n > 0, "bad arrays");
  float *out[4] = {in_mean, in_std, out_mean, out_std};
  m->net.moments(x, t, n, wide, out, row_squares);
  MLP_END
}

int cacg_mlp_set_normalization(cacg_mlp m, const float *in_mean, const float *in_std,
                               const float *out_mean, const float *out_std, double force_scale) {
  MLP_BEGIN
  need(in_mean && in_std && out_mean && out_std && force_scale > 0, "bad normalization");
  for (int i = 0; i < MLP_IN; i++) {
    need(in_std[i] > 0, "input std must be positive");
    m->net.norm[i] = in_mean[i];
    m->net.norm[MLP_IN + i] = 1.f / in_std[i];
  }
  for (int i = 0; i < MLP_OUT; i++) {
    need(out_std[i] > 0, "output std must be positive");
    m->net.norm[2 * MLP_IN + i] = out_mean[i];
    m->net.norm[2 * MLP_IN + MLP_OUT + i] = out_std[i];
  }
  m->net.force_scale = force_scale;
  m->net.upload_norm();
  m->net.sync();
  MLP_END
}

int cacg_mlp_get_normalization(cacg_mlp m, float *in_mean, float *in_std, float *out_mean,
                               float *out_std, double *force_scale) {
  MLP_BEGIN
  for (int i = 0; i < MLP_IN; i++) {
    if (in_mean) in_mean[i] = m->net.norm[i];
    if (in_std) in_std[i] = 1.f / m->net.norm[MLP_IN + i];
  }
  for (int i = 0; i < MLP_OUT; i++) {
    if (out_mean) out_mean[i] = m->net.norm[2 * MLP_IN + i];
    if (out_std) out_std[i] = m->net.norm[2 * MLP_IN + MLP_OUT + i];
  }
  if (force_scale) *force_scale = m->net.force_scale;
  MLP_END
}

int cacg_mlp_loss_grad(cacg_mlp m, int member, const float *x, const float *t, int n,
                       double *loss, float *grad) {
  MLP_BEGIN
  Net &N = m->net;
  need(x && t && n > 0 && member >= 0 && member < N.members, "bad arguments");
  const int B = (n + 127) / 128 * 128, tiles = B / 128;
  upload_set(N, x, t, n);
  const cacg::gemm::TrainArgs ta = N.batch(member, 1, B, n);
  N.loss.ensure(tiles, N.stream);
  Plan plan(ta);
  N.gather(ta, N.xf.p, N.tf.p, nullptr, 0, n);
  cacg::gemm::train_passes(*plan.p, N.loss.p, N.stream);
  N.gradients(ta, member);
  std::vector<double> h(tiles);
  cacg::check(cudaMemcpyAsync(h.data(), N.loss.p, sizeof(double) * tiles, cudaMemcpyDeviceToHost, N.stream), "loss");
  N.check_err();
  double l = 0.0;
  for (double q : h) l += q;
  if (loss) *loss = l / ((double) n * MLP_OUT);
  if (grad) {
    cacg::check(cudaMemcpyAsync(grad, N.g.p + (size_t) member * kNParam, sizeof(float) * kNParam,
                                cudaMemcpyDeviceToHost, N.stream), "grad");
    N.sync();
  }
  N.trim();
  MLP_END
}

int cacg_mlp_train(cacg_mlp m, const float *x, const float *t, long long n, int epochs, int batch,
                   float lr, unsigned long long seed, double *epoch_loss) {
  MLP_BEGIN
  Net &N = m->net;
  need(x && t && epochs > 0 && batch >= 128 && batch % 128 == 0 && n >= batch && lr > 0,
       "bad training arguments (batch a positive multiple of 128, n >= batch)");
  const long long nbatch = n / batch;  // whole batches only
  const int members = N.members, tiles = batch / 128;
  // the shuffles of an epoch, member by member from one random sequence: each
  // takes n - 1 numbers, so every shuffle's place in the sequence is known, and
  // the members' are made side by side, the next epoch's while this one runs
  std::vector<std::vector<int>> perm[2];
  for (auto &e : perm) e.assign(members, std::vector<int>(n));
  auto shuffle = [&](int ep, int k) {
    std::vector<int> &q = perm[ep & 1][k];
    cacg::mlp::Rng rng{seed};
    rng.skip((unsigned long long) ((long long) ep * members + k) * (unsigned long long) (n - 1));
    for (long long i = 0; i < n; i++) q[i] = (int) i;
    for (long long i = n - 1; i > 0; i--) std::swap(q[i], q[rng.next() % (unsigned long long) (i + 1)]);
  };
  Workers workers;
  auto start = [&](int ep) {
    for (int k = 0; k < members; k++) workers.run([&shuffle, ep, k] { shuffle(ep, k); });
  };
  start(0);
  upload_set(N, x, t, n);
  // All members at a time fill the SMs at usual batches; their arrays take 10 KB a row and
  // member, so with batches of millions of rows as many at a time as the device has room for
  // (a member's step needs nothing of the others').
  int at_once = members;
  while (true) {
    try {
      N.batch(0, at_once, batch, batch);
      break;
    } catch (const CudaError &e) {
      if (e.code != cudaErrorMemoryAllocation || at_once == 1) throw;
      cudaGetLastError();
      N.release_batch();
      at_once = (at_once + 1) / 2;
    }
  }
  N.loss.ensure((size_t) nbatch * members * tiles, N.stream);
  struct Group {
    int first;
    cacg::gemm::TrainArgs ta;
    std::unique_ptr<Plan> plan;
  };
  std::vector<Group> groups;
  for (int k = 0; k < members; k += at_once) {
    const cacg::gemm::TrainArgs ta = N.batch(k, std::min(at_once, members - k), batch, batch);
    groups.push_back({k, ta, std::unique_ptr<Plan>(new Plan(ta))});
  }
  cacg::DBuf<int> didx;
  const long long istride = batch * nbatch;
  didx.ensure((size_t) istride * members, N.stream);
  for (int ep = 0; ep < epochs; ep++) {
    // cosine schedule from lr to lr/20
    const float lr_ep = (float) (lr * (0.05 + 0.95 * 0.5 * (1 + std::cos(M_PI * ep / epochs))));
    workers.wait();
    for (int k = 0; k < members; k++)
      cacg::check(cudaMemcpyAsync(didx.p + k * istride, perm[ep & 1][k].data(), sizeof(int) * istride,
                                  cudaMemcpyHostToDevice, N.stream), "perm");
    if (ep + 1 < epochs) start(ep + 1);  // into the other buffers
    for (long long b = 0; b < nbatch; b++)
      for (const Group &q : groups) {
        N.gather(q.ta, N.xf.p, N.tf.p, didx.p + q.first * istride + b * batch, istride, batch);
        cacg::gemm::train_passes(*q.plan->p, N.loss.p + ((size_t) b * members + q.first) * tiles,
                                 N.stream);
        N.adam(q.ta, q.first, lr_ep);
      }
    N.sync();  // the shuffles' buffers are reused two epochs on
    N.adam_steps += nbatch;
  }
  if (epoch_loss) {
    std::vector<double> h((size_t) nbatch * members * tiles);
    cacg::check(cudaMemcpyAsync(h.data(), N.loss.p, sizeof(double) * h.size(), cudaMemcpyDeviceToHost,
                                N.stream), "loss");
    N.sync();
    double lsum = 0.0;
    for (int k = 0; k < members; k++)
      for (long long b = 0; b < nbatch; b++) {
        double l = 0.0;
        for (int q = 0; q < tiles; q++) l += h[((size_t) b * members + k) * tiles + q];
        lsum += l / ((double) batch * MLP_OUT);
      }
    *epoch_loss = lsum / (double) (members * nbatch);
  }
  N.check_err();
  N.trim();
  didx.release();
  MLP_END
}

int cacg_mlp_predict(cacg_mlp m, const float *x, long long n, float *mean, float *spread) {
  MLP_BEGIN
  Net &N = m->net;
  need(x && n > 0 && (mean || spread), "bad arguments");
  upload_set(N, x, nullptr, n);
  N.dm.ensure((size_t) n * MLP_OUT, N.stream);
  N.ds.ensure((size_t) n, N.stream);
  N.ensure_err(N.stream);
  N.predict_device(N.xf.p, n, N.dm.p, N.ds.p, N.stream);
  if (mean)
    cacg::check(cudaMemcpyAsync(mean, N.dm.p, sizeof(float) * n * MLP_OUT, cudaMemcpyDeviceToHost, N.stream), "mean");
  if (spread)
    cacg::check(cudaMemcpyAsync(spread, N.ds.p, sizeof(float) * n, cudaMemcpyDeviceToHost, N.stream), "spread");
  N.check_err();  // waits for the copies too
  N.trim();
  MLP_END
}

int cacg_gemm_bf16_tn(const void *a, int lda, const void *b, int ldb, float *c, int ldc, int m_,
                      int n_, int k_, int *err, void *stream) {
  if (!a || !b || !c || !err || m_ <= 0 || n_ <= 0 || k_ <= 0 || ldc < n_) return CACG_EINVAL;
  try {
    cacg::gemm::gemm_tn(a, lda, b, ldb, m_, n_, k_, c, ldc, err, static_cast<cudaStream_t>(stream));
  } catch (const CudaError &e) {
    return e.code == cudaErrorInvalidValue ? CACG_EINVAL : CACG_ECUDA;
  }
  return CACG_OK;
}

}  // extern "C"
