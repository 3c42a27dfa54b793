// FP64 atom passes (sm_103a): one block per 8 atoms.
//
// Included by k_force_exact.cu (FP64_EXACT_TU, -fmad=false: the reference's
// sequence of IEEE operations per pair and its order of summation, bit for
// bit) and k_force_fma.cu, after the helpers of elem_fp64.cuh.  The
// arithmetic follows PairLJCut::compute (pair_lj_cut.cpp:227-288) and
// PairEAM::compute (pair_eam.cpp:584-746).
//
// What bounds it: the FP64 unit in large systems, the chain of one thread's
// pairs in small ones (a thread per atom leaves 16,384 atoms on 3 warps per
// SM).  A block's warps scan the lists of 8 consecutive atoms, 32 entries at a
// time, with the FP32 test on the float copies, and buffer what passes in list
// order; all threads evaluate the buffered pairs (full warps), and one thread
// per atom and component adds the terms in list order.  The density pass
// leaves the short list and each pair's r (and 1/r with contraction) for the
// force pass, which then has no distance, cutoff or square root to form: 17
// of its 65 FP64 instructions per pair.  Without contraction, the squared distance
// and the splines are formed by the integer units (soft_fp64.cuh; the FP64 unit does
// 20 of 31 instructions a pair in the density pass, 30 of 44 in the force pass):
// 266,200 atoms 854 -> 594 and 1,199 -> 819 us, the FP64 unit still busy 84 %; LJ, 16,384
// atoms, 86 -> 68 us.  The distances take 8 or 16 bytes a list entry, more than the lists;
// where the device has no room for them (from some 80 M atoms on) the force pass forms them
// again, the same bits (STORED false).
#pragma once
#include "internal.h"

namespace cacg {
namespace FP64NS {

namespace {

constexpr int AB = 8;           // atoms per block
constexpr int ATOM_CAP = 96;    // buffered entries per atom and round
// Threads per block of a pass.  (The force pass with contraction waits on its loads,
// 70 % FP64 unit: 247,808 atoms 743 us with 128 threads, 628 with 64; the others, 84 %
// FP64 unit, get slower, 664 -> 683 and 819 -> 869 us.)
__host__ __device__ constexpr int atom_nt(int pass) {
#ifdef FP64_EXACT_TU
  return 128;
#else
  return pass == 2 ? 64 : 128;
#endif
}

#ifdef FP64_EXACT_TU
using PairR = double;           // r; negative: outside the cutoff
#else
using PairR = double2;          // r, 1/r
#endif

__device__ __forceinline__ float rsq_f32(float4 a, float4 b) {
  const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
  return dx * dx + dy * dy + dz * dz;
}

#ifdef FP64_EXACT_TU
// a spline's cubic, or its derivative's quadratic, by the integer units
// (spline_value, spline_deriv: N = 3, 2 Horner steps)
template <int N>
__device__ __forceinline__ double soft_spline(const double *__restrict__ c, const soft::Op &p) {
  auto op = [&](int k) {
    const double v = c[k];
    return soft::op_of((unsigned) __double2hiint(v), (unsigned) __double2loint(v));
  };
  constexpr int first = N == 3 ? 3 : 0;
  soft::Acc s = soft::add(soft::mul(op(first), p), soft::acc_of(op(first + 1)));
#pragma unroll
  for (int k = 2; k <= N; k++)
    s = soft::add(soft::mul(soft::op_of(s), p), soft::acc_of(op(first + k)));
  return __longlong_as_double((long long) soft::bits(s));
}

// dx^2 + dy^2 + dz^2 by the integer units
__device__ __forceinline__ double soft_rsq(double dx, double dy, double dz) {
  const unsigned hx = (unsigned) __double2hiint(dx), lx = (unsigned) __double2loint(dx);
  const unsigned hy = (unsigned) __double2hiint(dy), ly = (unsigned) __double2loint(dy);
  const unsigned hz = (unsigned) __double2hiint(dz), lz = (unsigned) __double2loint(dz);
  if (!soft::dot_ready(hx, lx) || !soft::dot_ready(hy, ly) || !soft::dot_ready(hz, lz))
    return dx * dx + dy * dy + dz * dz;
  soft::Op o = soft::op_of(hx, lx);
  soft::Acc s = soft::mul(o, o);
  o = soft::op_of(hy, ly);
  s = soft::add(s, soft::mul(o, o));
  o = soft::op_of(hz, lz);
  s = soft::add(s, soft::mul(o, o));
  return __longlong_as_double((long long) soft::bits(s));
}
#endif

#ifndef FP64_EXACT_TU
__device__ __forceinline__ double2 pair_r(double rsq) {
  const double recip = rsqrt_nr(rsq);
  return make_double2(rsq * recip, recip);
}
#else
__device__ __forceinline__ double pair_r(double rsq) { return sqrt(rsq); }
#endif

__device__ __forceinline__ double pair_rsq(double dx, double dy, double dz) {
#ifdef FP64_EXACT_TU
  return soft_rsq(dx, dy, dz);
#else
  return dx * dx + dy * dy + dz * dz;
#endif
}

// PASS 0: LJ forces; 1: EAM densities and F'(rho); 2: EAM forces from the
// short lists and distances (STORED) of pass 1
template <int PASS, bool STORED>
__global__ void __launch_bounds__(atom_nt(PASS))
k_atoms64(Atoms64Args a, EamTables e, const LJTab *__restrict__ tab) {
  constexpr int ATOM_NT = atom_nt(PASS);
  constexpr int NC = PASS == 1 ? 1 : NT3;   // buffered values per pair
  constexpr int NS = PASS == 1 ? 1 : 3;     // sums per atom
  __shared__ double s_t[AB][NC][ATOM_CAP + 1];
  __shared__ int s_ent[PASS == 2 ? 1 : AB][ATOM_CAP];
  __shared__ int s_cnt[AB], s_at[AB], s_len[AB], s_base[AB];
  __shared__ double4 s_x[AB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = blockIdx.x * AB, nb = min(AB, a.nlocal - i0);
  if (tid < AB) {
    s_cnt[tid] = s_at[tid] = s_base[tid] = s_len[tid] = 0;
    if (tid < nb) {
      s_x[tid] = a.x[i0 + tid];
      s_len[tid] = PASS == 2 ? a.snum[i0 + tid] : a.num[i0 + tid];
    }
  }
  const int my = tid % AB, i = i0 + my;
  const int ti = PASS == 0 && my < nb ? a.type[i] * (MAXT + 1) : 0;
  const double fpi = PASS == 2 && my < nb ? a.fp[i] : 0.0;
  double acc = 0.0;  // threads below NS * nb: atom tid / NS, component tid % NS
  __syncthreads();
  while (true) {
    // the next entries of each atom: what passes the FP32 test, in list order
    // (pass 2: the short list itself)
    if (PASS == 2) {
      if (tid < nb) {
        s_cnt[tid] = min(s_len[tid] - s_at[tid], ATOM_CAP);
        s_at[tid] += s_cnt[tid];
      }
    } else {
      for (int r = warp; r < nb; r += ATOM_NT / 32) {
        const int n = s_len[r];
        const float4 hi = a.xh[i0 + r];
        const int *__restrict__ list = a.list + i0 + r;
        int at = s_at[r], cnt = 0;
        for (; at < n && cnt + 32 <= ATOM_CAP; at += 32) {
          int j = 0;
          bool pass = false;
          if (at + lane < n) {
            j = __ldg(list + (size_t) (at + lane) * a.stride);
            pass = rsq_f32(hi, __ldg(a.xh + j)) <= a.cut_pass;
          }
          const unsigned b = __ballot_sync(0xffffffffu, pass);
          if (pass) s_ent[r][cnt + __popc(b & ((1u << lane) - 1u))] = j;
          cnt += __popc(b);
        }
        __syncwarp();
        if (lane == 0) {
          s_cnt[r] = cnt;
          s_at[r] = min(at, n);
        }
      }
    }
    __syncthreads();
    bool more = false;
#pragma unroll
    for (int r = 0; r < AB; r++) more = more || s_at[r] < s_len[r];
    // the pairs, the 8 atoms side by side (whole sectors of the short lists)
    const int cnt = s_cnt[my];
    if (cnt > 0) {
      const double4 xi = s_x[my];
      const size_t first = (size_t) s_base[my] * a.stride + i;
      for (int k = tid / AB; k < cnt; k += ATOM_NT / AB) {
        const size_t at = first + (size_t) k * a.stride;
        const int j = PASS == 2 ? __ldg(a.slist + at) : s_ent[PASS == 2 ? 0 : my][k];
        const double4 xj = a.x[j];
        const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        double fpair = 0.0;
        bool in;
        if (PASS == 2) {
          PairR pr;
          if (STORED) {
            pr = reinterpret_cast<const PairR *>(a.sr)[at];
          } else {
            const double rsq = pair_rsq(dx, dy, dz);
            in = rsq < e.cutforcesq;
            pr = pair_r(rsq);
          }
#ifdef FP64_EXACT_TU
          const double r = pr;
#else
          const double r = pr.x;
#endif
          if (STORED) in = !(r < 0.0);
          if (in) {
            double p;
            const int m = split_index(r * e.rdr + 1.0, e.nr - 1, p);
            const double *c = e.rhor + 7 * (size_t) m;
            const double *z = e.z2r + 7 * (size_t) m;
#ifdef FP64_EXACT_TU
            double rhoip, z2p, z2;
            if (e.soft) {
              const soft::Op q = soft::op_of((unsigned) __double2hiint(p), (unsigned) __double2loint(p));
              rhoip = soft_spline<2>(c, q);
              z2p = soft_spline<2>(z, q);
              z2 = soft_spline<3>(z, q);
            } else {
              rhoip = spline_deriv(c, p);
              z2p = spline_deriv(z, p);
              z2 = spline_value(z, p);
            }
            const double recip = 1.0 / r;
#else
            const double rhoip = spline_deriv(c, p);
            const double z2p = spline_deriv(z, p);
            const double z2 = spline_value(z, p);
            const double recip = pr.y;
#endif
            const double phi = z2 * recip;
            const double phip = z2p * recip - phi * recip;
            // one table for every type pair (single funcfl file)
            const double psip = fpi * rhoip + __ldg(a.fp + j) * rhoip + phip;
            fpair = -psip * recip;
          }
        } else {
          const double rsq = pair_rsq(dx, dy, dz);
          const int ij = PASS == 0 ? ti + a.type[j] : 0;
          in = rsq < (PASS == 0 ? tab->cutsq[ij] : e.cutforcesq);
          if (PASS == 0) {
            if (in) {
#ifdef FP64_EXACT_TU
              const double r2inv = 1.0 / rsq;
#else
              const double r2inv = rcp_nr(rsq);
#endif
              const double r6inv = r2inv * r2inv * r2inv;
              const double forcelj = r6inv * (tab->lj1[ij] * r6inv - tab->lj2[ij]);
              fpair = forcelj * r2inv;
            }
          } else {
            double t = 0.0;
            PairR pr;
#ifdef FP64_EXACT_TU
            pr = -1.0;
#else
            pr = make_double2(-1.0, 0.0);
#endif
            if (in) {
              pr = pair_r(rsq);
#ifdef FP64_EXACT_TU
              const double r = pr;
#else
              const double r = pr.x;
#endif
              double p;
              const int m = split_index(r * e.rdr + 1.0, e.nr - 1, p);
#ifdef FP64_EXACT_TU
              if (e.soft)
                t = soft_spline<3>(e.rhor + 7 * (size_t) m,
                                   soft::op_of((unsigned) __double2hiint(p), (unsigned) __double2loint(p)));
              else
#endif
                t = spline_value(e.rhor + 7 * (size_t) m, p);
            }
            s_t[my][0][k] = t;
            a.slist[at] = j;
            if (STORED) reinterpret_cast<PairR *>(a.sr)[at] = pr;
          }
        }
        if (PASS != 1) {
          // a pair beyond the cutoff leaves zeros, which change no sum
#ifdef FP64_EXACT_TU
          s_t[my][0][k] = in ? dx * fpair : 0.0;
          s_t[my][1 % NC][k] = in ? dy * fpair : 0.0;
          s_t[my][2 % NC][k] = in ? dz * fpair : 0.0;
#else
          s_t[my][0][k] = in ? dx : 0.0;
          s_t[my][1 % NC][k] = in ? dy : 0.0;
          s_t[my][2 % NC][k] = in ? dz : 0.0;
          s_t[my][3 % NC][k] = fpair;
#endif
        }
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
      for (int k = 0; k < n; k++) acc = PASS == 1 ? acc + t[k] : fma(t[k], g[k], acc);
#endif
    }
    if (!more) break;
    __syncthreads();
    if (tid < AB) {
      s_base[tid] += s_cnt[tid];
      s_cnt[tid] = 0;
    }
    __syncthreads();
  }
  if (PASS == 1) {
    if (tid < nb) {
      a.snum[i0 + tid] = s_base[tid] + s_cnt[tid];
      a.rho[i0 + tid] = acc;
      a.fp[i0 + tid] = eam_slope(e, acc);
    }
  } else {
    if (PASS == 0 && tid < nb) a.snum[i0 + tid] = s_base[tid] + s_cnt[tid];
    if (tid < 3 * nb) a.f[3 * (size_t) i0 + tid] = acc;
  }
}

}  // namespace

// pass 0: LJ forces; 1: EAM densities, F'(rho), short lists; 2: EAM forces
void atom_pass(const Atoms64Args &a, int pass, const EamTables &e, const void *ljtab, cudaStream_t s) {
  if (a.nlocal <= 0) return;
  auto k = pass == 0   ? k_atoms64<0, false>
           : pass == 1 ? (a.sr ? k_atoms64<1, true> : k_atoms64<1, false>)
                       : (a.sr ? k_atoms64<2, true> : k_atoms64<2, false>);
  k<<<(a.nlocal + AB - 1) / AB, atom_nt(pass), 0, s>>>(a, e, (const LJTab *) ljtab);
  check(cudaGetLastError(), "atom_pass");
}

// bytes that a pair's distance takes between passes 1 and 2
size_t pair_bytes() { return sizeof(PairR); }

}  // namespace FP64NS (per translation unit)
}  // namespace cacg
