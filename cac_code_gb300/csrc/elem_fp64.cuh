// FP64 element passes (sm_103a): one block per element, positions of only the
// sites a row interacts with.
//
// Included by two translation units, like force_fp64.cuh: k_force_exact.cu
// (-fmad=false, FP64_EXACT_TU) keeps the reference's sequence of IEEE
// operations per pair and its order of summation, so its results are bit for
// bit the reference's; k_force_fma.cu contracts and uses the refined
// reciprocals.  The arithmetic follows PairLJCut::ecompute
// (pair_lj_cut.cpp:295-442), PairEAM::ecompute (pair_eam.cpp:761-1141) and the
// gather of pair_lj_cut.cpp:424-428.
//
// What bounds it: the FP64 unit (a warp instruction holds it for 16 cycles).
// An interpolated position costs 45 FP64 instructions, and of the 1,331 sites
// of an 11 x 11 x 11 element the rows of 2 x 2 x 2 Gauss points and 8 nodes
// reach about 500.  So each row's list is tested in FP32 first, on coordinates
// relative to the element's node 0 with a bound derived from their size
// (pass_limit), and only the entries that pass get an FP64 position, formed
// where the pair is evaluated: no site array, no list of the step in memory,
// no F'(rho) of sites that nothing reaches.  And the positions, with the densities of
// the sites where they are not contracted, come from the integer units
// (soft_fp64.cuh), which are idle otherwise: the FP64 unit is left 53 of 98
// instructions a pair.  64,000 elements with contraction: forces 5,084 -> 3,230 us, the
// FP64 unit busy 74 % of it and the ALU 67 %, densities 1,122 -> 925 us (ALU 77 %); 7,200
// without: forces 1,113 -> 690 us.
//
// A block takes RB rows at a time.  Its warps scan the rows' lists 32 entries
// at a time and append what passes, in list order, to the rows' buffers in
// shared memory; all threads then evaluate the buffered pairs of all rows
// (full warps whatever a row holds), leave each pair's terms in shared memory,
// and one thread per row and component adds them in list order.  Rows whose
// buffer fills up go on where they stopped in a further round.
#pragma once
#include "internal.h"
#include "soft_fp64.cuh"
#include <type_traits>

namespace cacg {
namespace FP64NS {

namespace {

constexpr int RB = 8;           // rows of an element per round
constexpr int ROW_CAP = 96;     // buffered entries per row
constexpr int ELEM_NT = 128;    // threads per block
constexpr int FEW_NT = 256, FEW_CL = 4;  // with few elements: threads, or blocks an element

#ifdef FP64_EXACT_TU
constexpr int NT3 = 3;          // buffered per pair: the three terms
constexpr bool SOFT_RHO = true; // a site's density by the integer units as well
#else
constexpr int NT3 = 4;          // the vector and the pair factor (summed with one FMA)
constexpr bool SOFT_RHO = false;  // (contracted here)
#endif

// m = min((int) q, n1) and p = min(q - m, 1): for 1 <= q < 2^20 from the bits
// of q, without conversions (they issue at the FP64 rate): the integer part is
// q with the mantissa bits below the point cleared.  m is at least 1, as it is
// for every r >= 0 and as rho's index is clamped.
__device__ __forceinline__ int split_index(double q, int n1, double &p) {
  const int hi = __double2hiint(q);
  const unsigned e = (unsigned) (hi >> 20) - 1023u;
  if (e < 20u) {
    const int sh = 20 - (int) e;
    const int m = ((hi & 0xFFFFF) | 0x100000) >> sh;
    if (m <= n1) {
      p = q - __hiloint2double(hi & (int) (0xFFFFFFFFu << sh), 0);
      return m;
    }
  }
  int m = (int) q;
  m = m < n1 ? m : n1;
  m = m > 1 ? m : 1;
  p = q - m;
  p = p < 1.0 ? p : 1.0;
  return m;
}

// FP32 limit of the squared distance of two points of an element (coordinates
// relative to node 0, at most R; absolute coordinates at most X) that FP64
// arithmetic may place within the cutoff.  With u = 2^-24 a relative node is
// within u R of its value, an interpolated coordinate within 10 u R (weights
// >= 0 of sum 1, rounded once, eight products and sums), a difference within
// 22 u R; FP64 positions are within 12 * 2^-53 X each.  Both bounds are taken
// with slack, and the sum of squares and the limit itself within 1e-5.
__device__ __forceinline__ float pass_limit(float cutsq, float R, float X) {
  const float u = 5.9604645e-8f, v = 1.110223e-16f;
  const float r = sqrtf(cutsq) * 1.000001f + 1.7320509f * (24.f * u * R + 32.f * v * X);
  return r * r * 1.00001f;
}

// w0 x0 + w1 x1 + ... over an element's 8 nodes without contraction in either
// mode, as the reference interpolates (its first addition, to 0, changes
// nothing but the sign of a zero).  Coordinates reach 1e3 and more: a fused
// rounding would move a site by ~1e-13, which the stiff pair forces amplify.
__device__ __forceinline__ double node_sum(const double (&w)[NPE], const double *__restrict__ x,
                                           int stride) {
  double a = __dmul_rn(w[0], x[0]);
#pragma unroll
  for (int k = 1; k < NPE; k++) a = __dadd_rn(a, __dmul_rn(w[k], x[stride * k]));
  return a;
}

__device__ __forceinline__ void load8(const double *__restrict__ p, double (&w)[NPE]) {
#pragma unroll
  for (int k = 0; k < NPE / 2; k++) {
    const double2 d = __ldg(reinterpret_cast<const double2 *>(p) + k);
    w[2 * k] = d.x;
    w[2 * k + 1] = d.y;
  }
}

__device__ __forceinline__ double eam_slope(const EamTables &e, double rho) {
  double p;
  const int m = split_index(rho * e.rdrho + 1.0, e.nrho - 1, p);
  const double *c = e.frho + 7 * (size_t) m;
  return (c[0] * p + c[1]) * p + c[2];
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// *p of the cluster's first block
__device__ __forceinline__ void store_first(double *p, double v) {
  unsigned a = (unsigned) __cvta_generic_to_shared(p);
  asm volatile("{\n .reg .u32 r;\n mapa.shared::cluster.u32 r, %0, 0;\n st.shared::cluster.f64 [r], %1;\n}"
               ::"r"(a), "d"(v) : "memory");
}

// the sums of the weights times N groups of 8 operands (x, y, z, then the densities)
template <int N>
__device__ __forceinline__ void soft_dots(const double (&w)[NPE], const soft::Op *s_op, double &x,
                                          double &y, double &z, double &rho) {
  soft::Op o[NPE];
  x = y = z = rho = 0.0;
#pragma unroll
  for (int k = 0; k < NPE; k++)
    o[k] = soft::op_of((unsigned) __double2hiint(w[k]), (unsigned) __double2loint(w[k]));
#pragma unroll 1
  for (int d = 0; d < N; d++) {
    soft::Acc s = soft::mul(o[0], s_op[8 * d]);
#pragma unroll
    for (int k = 1; k < NPE; k++) s = soft::add(s, soft::mul(o[k], s_op[8 * d + k]));
    const double v = __longlong_as_double((long long) soft::bits(s));
    x = y;
    y = z;
    if (N == 4) {
      z = rho;
      rho = v;
    } else {
      z = v;
    }
  }
}

// DENSITY: the 8 node rows of each element -> erho; otherwise the force rows
// (row list fjj of the type; all rows when it is null) -> nodef.
// SELF: every list entry is a site of the row's own element.
// FEW: with few elements a block has an SM's FP64 unit to itself or SMs are idle.  2:
// twice the threads and no integer arithmetic; 1: a cluster of FEW_CL blocks per element
// instead, two rows of a round each, whose forces the first block gathers from its shared
// memory.  EAM forces in the exact mode alone, us, with FEW 1 / 2 / 0: 64 elements 31 / 37 /
// 51, 128 45 / 37 / 52, 256 84 / 56 / 63, 512 164 / 106 / 78; LJ 12 / 16 / 21, 16 / 16 / 21, 30
// / 23 / 24, 57 / 42 / 32.  Beside the atom passes, which share the FP64 units, a run: 32
// elements and 1,024 atoms 706 / 877 / 912, 64 and 16,384 1,885 / 1,719 / 1,838, 128 and 23,232
// 3,994 / 3,746 / 3,695, 256 and 23,232 4,839 / 4,219 / 3,872: 1 where the atoms' blocks leave
// SMs idle, 2 up to an element an SM.
template <bool EAM, bool DENSITY, bool SELF, int FEW>
__global__ void __launch_bounds__(FEW == 2 ? FEW_NT : ELEM_NT, FEW == 2 ? 2 : FEW ? 4 : 7)
k_elem64(Elem64Args a, EamTables eam, double lj1, double lj2, double cutsq,
         double *__restrict__ out) {
  constexpr int NC = DENSITY ? 1 : NT3, NS = DENSITY ? 1 : 3;  // buffered values, sums
  constexpr int ELEM_NT = FEW == 2 ? FEW_NT : FP64NS::ELEM_NT;
  constexpr bool SOFT = SELF && FEW == 0, CL = FEW == 1;
  __shared__ double s_nx[24], s_er[NPE], s_p[RB][3], s_N[RB][NPE], s_fpi[RB], s_f[RB][3];
  __shared__ double s_t[RB][NC][ROW_CAP + 1];
  __shared__ int s_ent[RB][ROW_CAP];
  __shared__ int s_cnt[RB], s_at[RB], s_len[RB], s_start[RB], s_jj[RB];
  __shared__ float4 s_nf4[6];
  __shared__ float s_pf[RB][3];
  __shared__ float s_lim;
  // by the integer units (soft_fp64.cuh): the nodes' coordinates by axis, then their
  // densities; whether all of them can be
  constexpr int NDOT = SOFT_RHO && EAM && !DENSITY ? 4 : 3;
  __shared__ soft::Op s_op[SOFT ? 8 * NDOT : 1];
  __shared__ int s_hard;
  float *s_nf = reinterpret_cast<float *>(s_nf4);
  if (CL && !DENSITY) cluster_sync();  // the first block runs before others store to it
  // (a cluster: the gather's rows, of all blocks)
  __shared__ double s_gN[CL && !DENSITY ? RB : 1][NPE];
  __shared__ int s_gj[CL && !DENSITY ? RB : 1];
  const int rank = CL ? (int) blockIdx.x % FEW_CL : 0;
  const int e = CL ? (int) blockIdx.x / FEW_CL : (int) blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = a.etype[e], ioff = a.int_off[ty];
  const int naz = a.nae[3 * ty + 2];
  const double *__restrict__ S0 = a.spa_inter + (size_t) a.inter_off[ty] * NPE;
  const float4 *__restrict__ F0 = a.spa_inter_f + (size_t) a.inter_off[ty] * 2;
  const int kb = a.kb, kmask = (1 << kb) - 1;
  if (SOFT) {
    if (tid == 0) s_hard = !a.soft;
    __syncthreads();
  }
  if (warp == 0) {
    float r = 0.f, x = 0.f;
    if (lane < 24) {
      const double v = a.nodex[24 * (size_t) e + lane];
      s_nx[lane] = v;
      if (SOFT) {
        const unsigned h = (unsigned) __double2hiint(v), l = (unsigned) __double2loint(v);
        s_op[lane % 3 * 8 + lane / 3] = soft::op_of(h, l);
        if (!soft::dot_ready(h, l)) s_hard = 1;
      }
      const double v0 = __shfl_sync(0x00FFFFFFu, v, lane % 3);
      const float f = SELF ? (float) (v - v0) : (float) v;
      s_nf[lane] = f;
      r = fabsf(f);
      x = fabsf((float) v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
      x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    }
    if (lane == 0) s_lim = SELF ? pass_limit((float) cutsq, r, x) : a.cut_pass;
  } else if (warp == 1 && EAM && !DENSITY) {
    if (lane < NPE) {
      const double v = a.erho[NPE * (size_t) e + lane];
      s_er[lane] = v;
      if (SOFT && NDOT == 4) {
        const unsigned h = (unsigned) __double2hiint(v), l = (unsigned) __double2loint(v);
        s_op[SOFT ? 8 * (NDOT - 1) + lane : 0] = soft::op_of(h, l);
        if (!soft::dot_ready(h, l)) s_hard = 1;
      }
    }
  }
  const int nr_rows = DENSITY ? NPE : (a.fjj ? a.fjj_off[ty + 1] - a.fjj_off[ty] : a.numint[ty]);
  double nf = 0.0;  // threads 0..23: the nodal force component
  for (int rb = 0; rb < nr_rows; rb += RB) {
    const int all = min(RB, nr_rows - rb), lo = CL ? rank * (RB / FEW_CL) : 0;
    const int nb = CL ? max(0, min(RB / FEW_CL, all - lo)) : all;
    __syncthreads();
    if (CL && !DENSITY && rank == 0)
      for (int t = tid; t < all * NPE; t += ELEM_NT) {
        const int q = rb + t / NPE, jj = a.fjj ? a.fjj[a.fjj_off[ty] + q] : q;
        s_gN[CL && !DENSITY ? t / NPE : 0][t % NPE] = a.spa_int[((size_t) ioff + jj) * NPE + t % NPE];
        if (t % NPE == 0) s_gj[CL && !DENSITY ? t / NPE : 0] = jj;
      }
    if (tid < nb) {
      const int q = rb + lo + tid;
      const int jj = DENSITY ? a.node_list[ty * NPE + q] : (a.fjj ? a.fjj[a.fjj_off[ty] + q] : q);
      const int r = a.row_first[e] + jj;
      s_jj[tid] = jj;
      s_start[tid] = a.row_start[r];
      s_len[tid] = a.row_start[r + 1] - a.row_start[r];
      s_at[tid] = 0;
    }
    __syncthreads();
    // the rows' points: FP64 (a row's node itself in the density pass) and FP32
    for (int t = tid; t < nb * 3; t += ELEM_NT) {
      const int r = t / 3, d = t % 3;
      if (DENSITY) {
        s_p[r][d] = s_nx[3 * (rb + lo + r) + d];
        s_pf[r][d] = s_nf[3 * (rb + lo + r) + d];
        continue;
      }
      double w[NPE];
      load8(a.spa_int + ((size_t) ioff + s_jj[r]) * NPE, w);
      s_p[r][d] = node_sum(w, s_nx + d, 3);
      float pf = 0.f;
#pragma unroll
      for (int k = 0; k < NPE; k++) {
        if (d == 0) s_N[r][k] = w[k];
        pf += (float) w[k] * s_nf[3 * k + d];
      }
      s_pf[r][d] = pf;
      if (EAM && d == 0) {
        double rho = 0.0;
#pragma unroll
        for (int k = 0; k < NPE; k++) rho += w[k] * s_er[k];
        s_fpi[r] = eam_slope(eam, rho);
      }
    }
    double acc = 0.0;  // threads below NS * nb: row tid / NS, component tid % NS
    __syncthreads();
    const float lim = s_lim;
    while (true) {
      // scan: what passes the FP32 test, in list order
      for (int r = warp; r < nb; r += ELEM_NT / 32) {
        const int n = s_len[r];
        const int *__restrict__ ent = a.ent + s_start[r];
        const float px = s_pf[r][0], py = s_pf[r][1], pz = s_pf[r][2];
        int at = s_at[r], cnt = 0;
        for (; at < n && cnt + 32 <= ROW_CAP; at += 32) {
          const bool live = at + lane < n;
          const int code = live ? __ldg(ent + at + lane) : 0;
          bool pass = false;
          if (live) {
            int line = code >> kb;
            const float4 *x4 = s_nf4;
            if (SELF) {
              line -= e * a.maxlines;
            } else {
              const int j = line / a.maxlines;
              line -= j * a.maxlines;
              if (j != e) x4 = a.node_f + 6 * (size_t) j;
            }
            float x[24];
#pragma unroll
            for (int k = 0; k < 6; k++) {
              const float4 v = x4[k];
              x[4 * k] = v.x;
              x[4 * k + 1] = v.y;
              x[4 * k + 2] = v.z;
              x[4 * k + 3] = v.w;
            }
            const int nj = line * naz + (code & kmask);
            const float4 w0 = __ldg(F0 + 2 * (size_t) nj), w1 = __ldg(F0 + 2 * (size_t) nj + 1);
            const float w[NPE] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
            float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
            for (int k = 0; k < NPE; k++) {
              sx = __fmaf_rn(w[k], x[3 * k], sx);
              sy = __fmaf_rn(w[k], x[3 * k + 1], sy);
              sz = __fmaf_rn(w[k], x[3 * k + 2], sz);
            }
            const float dx = px - sx, dy = py - sy, dz = pz - sz;
            pass = dx * dx + dy * dy + dz * dz <= lim;
          }
          const unsigned b = __ballot_sync(0xffffffffu, pass);
          if (pass) s_ent[r][cnt + __popc(b & ((1u << lane) - 1u))] = code;
          cnt += __popc(b);
        }
        if (lane == 0) {
          s_cnt[r] = cnt;
          s_at[r] = at;
        }
      }
      __syncthreads();
      int total = 0;
      bool more = false;
      for (int r = 0; r < nb; r++) {
        total += s_cnt[r];
        more = more || s_at[r] < s_len[r];
      }
      // the buffered pairs of all rows, one after another
      for (int idx = tid; idx < total; idx += ELEM_NT) {
        int r = 0, k = idx;
        while (k >= s_cnt[r]) k -= s_cnt[r++];
        const int code = s_ent[r][k];
        int line = code >> kb, j = e;
        if (SELF) {
          line -= e * a.maxlines;
        } else {
          j = line / a.maxlines;
          line -= j * a.maxlines;
        }
        const int nj = line * naz + (code & kmask);
        double S[NPE];
        load8(S0 + (size_t) nj * NPE, S);
        double sx, sy, sz, srho = 0.0;
        const bool hard = !SOFT || s_hard;
        if (hard) {
          const double *x = SELF || j == e ? s_nx : a.nodex + 24 * (size_t) j;
          sx = node_sum(S, x, 3);
          sy = node_sum(S, x + 1, 3);
          sz = node_sum(S, x + 2, 3);
        } else {
          soft_dots<NDOT>(S, s_op, sx, sy, sz, srho);
        }
        const double dx = s_p[r][0] - sx, dy = s_p[r][1] - sy, dz = s_p[r][2] - sz;
        const double rsq = dx * dx + dy * dy + dz * dz;
        double t0 = 0.0, fpair = 0.0;
        const bool in = rsq < cutsq;
        if (in) {
          if (EAM) {
#ifdef FP64_EXACT_TU
            const double rr = sqrt(rsq);
#else
            const double recip = rsqrt_nr(rsq);
            const double rr = rsq * recip;
#endif
            double p;
            const int m = split_index(rr * eam.rdr + 1.0, eam.nr - 1, p);
            const double *c = eam.rhor + 7 * (size_t) m;
            if (DENSITY) {
              t0 = ((c[3] * p + c[4]) * p + c[5]) * p + c[6];
            } else {
              const double *er = SELF || j == e ? s_er : a.erho + NPE * (size_t) j;
              double rho = srho;
              if (hard || NDOT == 3) {
                rho = 0.0;
#pragma unroll
                for (int q = 0; q < NPE; q++) rho += S[q] * er[q];
              }
              const double fpj = eam_slope(eam, rho);
              const double rhoip = (c[0] * p + c[1]) * p + c[2];
              const double *z = eam.z2r + 7 * (size_t) m;
              const double z2p = (z[0] * p + z[1]) * p + z[2];
              const double z2 = ((z[3] * p + z[4]) * p + z[5]) * p + z[6];
#ifdef FP64_EXACT_TU
              const double recip = 1.0 / rr;
#endif
              const double phi = z2 * recip;
              const double phip = z2p * recip - phi * recip;
              const double psip = (s_fpi[r] + fpj) * rhoip + phip;
              fpair = -psip * recip;
            }
          } else {
#ifdef FP64_EXACT_TU
            const double r2inv = 1.0 / rsq;
#else
            const double r2inv = rcp_nr(rsq);
#endif
            const double r6inv = r2inv * r2inv * r2inv;
            const double forcelj = r6inv * (lj1 * r6inv - lj2);
            fpair = forcelj * r2inv;
          }
        }
        // a pair beyond the cutoff leaves zeros, which change no sum
        if (DENSITY) {
          s_t[r][0][k] = t0;
        } else {
#ifdef FP64_EXACT_TU
          s_t[r][0][k] = in ? dx * fpair : 0.0;
          s_t[r][1 % NC][k] = in ? dy * fpair : 0.0;
          s_t[r][2 % NC][k] = in ? dz * fpair : 0.0;
#else
          s_t[r][0][k] = in ? dx : 0.0;
          s_t[r][1 % NC][k] = in ? dy : 0.0;
          s_t[r][2 % NC][k] = in ? dz : 0.0;
          s_t[r][3 % NC][k] = fpair;
#endif
        }
      }
      __syncthreads();
      if (tid < NS * nb) {
        const int r = tid / NS, n = s_cnt[r];
        const double *t = s_t[r][tid % NS];
#ifdef FP64_EXACT_TU
#pragma unroll 8
        for (int k = 0; k < n; k++) acc += t[k];
#else
        const double *g = s_t[r][NC - 1];
#pragma unroll 8
        for (int k = 0; k < n; k++) acc = DENSITY ? acc + t[k] : fma(t[k], g[k], acc);
#endif
      }
      if (!more) break;
      __syncthreads();
    }
    if (DENSITY) {
      if (tid < nb) out[NPE * (size_t) e + rb + lo + tid] = acc;
    } else {
      if (tid < 3 * nb) {
        if (CL) store_first(&s_f[lo + tid / 3][tid % 3], acc);
        else s_f[tid / 3][tid % 3] = acc;
      }
      if (CL) cluster_sync();
      else __syncthreads();
      // the nodal gather in row order (rows of weight 0 add nothing)
      if (rank == 0 && tid < 24) {
        if (CL) {
          for (int r = 0; r < all; r++)
            nf += a.weight[ioff + s_gj[CL && !DENSITY ? r : 0]] *
                  s_gN[CL && !DENSITY ? r : 0][tid / 3] * s_f[r][tid % 3];
        } else {
          for (int r = 0; r < nb; r++)
            nf += a.weight[ioff + s_jj[r]] * s_N[r][tid / 3] * s_f[r][tid % 3];
        }
      }
      if (CL && rb + RB < nr_rows) cluster_sync();  // s_f is written again
    }
  }
  if (!DENSITY && rank == 0 && tid < 24) out[24 * (size_t) e + tid] = nf;
}

}  // namespace

#ifndef FP64_EXACT_TU
namespace {
__global__ void k_node_f(const double *__restrict__ nodex, long long n, float *__restrict__ out) {
  const long long t = blockIdx.x * (long long) blockDim.x + threadIdx.x;
  if (t < n) out[t] = (float) nodex[t];
}
}  // namespace

// float copies of all nodes, for lists that reach other elements
void node_floats(const double *nodex, int nelem, float4 *out, cudaStream_t s) {
  if (nelem <= 0) return;
  const long long n = 24LL * nelem;
  k_node_f<<<(int) ((n + 255) / 256), 256, 0, s>>>(nodex, n, reinterpret_cast<float *>(out));
  check(cudaGetLastError(), "node_floats");
}
#endif

void elem_pass(const Elem64Args &a, int pass, bool self, const EamTables &e, double lj1, double lj2,
               double cutsq, double *out, cudaStream_t s) {
  if (a.nlocal_e <= 0) return;
  auto pick = [&](auto few) {
    constexpr int FEW = decltype(few)::value;
    return pass == 0 ? (self ? k_elem64<false, false, true, FEW> : k_elem64<false, false, false, FEW>)
           : pass == 1 ? (self ? k_elem64<true, true, true, FEW> : k_elem64<true, true, false, FEW>)
                       : (self ? k_elem64<true, false, true, FEW> : k_elem64<true, false, false, FEW>);
  };
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (3LL * a.nlocal_e <= 2LL * nsm && a.natoms <= 8 * nsm) {
    cudaLaunchConfig_t c{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = FEW_CL;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    c.gridDim = dim3(FEW_CL * a.nlocal_e);
    c.blockDim = dim3(ELEM_NT);
    c.stream = s;
    c.attrs = at;
    c.numAttrs = 1;
    check(cudaLaunchKernelEx(&c, pick(std::integral_constant<int, 1>{}), a, e, lj1, lj2, cutsq, out),
          "elem_pass");
  } else if (a.nlocal_e <= nsm) {
    pick(std::integral_constant<int, 2>{})<<<a.nlocal_e, FEW_NT, 0, s>>>(a, e, lj1, lj2, cutsq, out);
  } else {
    pick(std::integral_constant<int, 0>{})<<<a.nlocal_e, ELEM_NT, 0, s>>>(a, e, lj1, lj2, cutsq, out);
  }
  check(cudaGetLastError(), "elem_pass");
}

}  // namespace FP64NS (per translation unit)
}  // namespace cacg
