// Neighbor lists on the device (sm_103a), compiled without FMA contraction so
// every distance predicate is the reference's own arithmetic:
//   * atom list: Neighbor::half_bin_no_newton (neighbor.cpp:546-625), a FULL list,
//     rsq <= cutneighmaxsq, j over stencil bins in stencil order and bin members
//     in index order -- so each row equals the reference's row entry for entry;
//   * element list: Neighbor::element_neighbor (element_neighbor.cpp:11-75) over
//     element centres with the same bins/stencil and rsq <= cut_allsq;
//   * integration-point list: Neighbor::node_neighbor (full_node_neighbor.cpp:19-239),
//     one warp per integration point; lanes test 32 lattice sites of a sub-element
//     at once and a ballot compacts the hits in the reference's site order.
// Lists are column-major (entry k of row i at k*stride + i) so that the force
// kernels, one thread per row, read them coalesced.
#include "ghosts.cuh"
#include "internal.h"

namespace cacg {

namespace {

inline int nblk(long long n, int t) { return (int) ((n + t - 1) / t); }

// Atom list, one warp per atom.  The stencil's bins that follow each other in
// x are one run of the bin-ordered members, so the warp walks the runs 32
// members at a time and a ballot appends the hits in the reference's order
// (stencil order, members in index order).  A distance is decided in FP32 on
// the float copies outside [lo, hi] (no float rounding moves a pair across the
// cutoff there) and in the reference's FP64 arithmetic inside: of ~560
// candidates a pair of FP64 units need not see more than the few in the band.
// The band is for coordinates up to a range; a member beyond it (an atom that left
// a box with fixed boundaries, or one near such an atom) has a NaN for a float
// coordinate (launch_gather_bin_x_atoms), so that neither side of the band takes it.
// One thread per atom with FP64 throughout took 1,133 us for 72,600 atoms.
constexpr int AL_BLOCK = 256;

__global__ void __launch_bounds__(AL_BLOCK)
k_atom_list(const double4 *__restrict__ x, const int *__restrict__ bin,
            const int *__restrict__ bstart, const float4 *__restrict__ bxf,
            const int2 *__restrict__ runs, int nruns, int mbins, int nlocal, double cutsq, float lo,
            float hi, int maxneigh, int stride, int *__restrict__ num, int *__restrict__ list,
            int *__restrict__ overflow) {
  const int i = (int) ((blockIdx.x * (long long) AL_BLOCK + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= nlocal) return;
  const double4 xi = x[i];
  const float fx = (float) xi.x, fy = (float) xi.y, fz = (float) xi.z;
  const int ib = bin[i];
  int n = 0;
  for (int r0 = 0; r0 < nruns; r0 += 32) {
    // this lane's run: its members' range
    int p0 = 0, p1 = 0;
    if (r0 + lane < nruns) {
      const int2 run = __ldg(runs + r0 + lane);
      const int b0 = max(ib + run.x, 0), b1 = min(ib + run.x + run.y, mbins);
      if (b0 < b1) {
        p0 = __ldg(bstart + b0);
        p1 = __ldg(bstart + b1);
      }
    }
    const int nr = min(32, nruns - r0);
    for (int r = 0; r < nr; r++) {
      const int q1 = __shfl_sync(0xffffffffu, p1, r);
      for (int q = __shfl_sync(0xffffffffu, p0, r); q < q1; q += 32) {
        bool hit = false;
        int j = i;
        if (q + lane < q1) {
          const float4 c = __ldg(bxf + q + lane);
          j = __float_as_int(c.w);
          const float gx = fx - c.x, gy = fy - c.y, gz = fz - c.z;
          const float g = gx * gx + gy * gy + gz * gz;
          hit = g < lo;
          if (!hit && !(g > hi)) {
            const double4 xj = x[j];
            const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
            hit = dx * dx + dy * dy + dz * dz <= cutsq;
          }
          hit = hit && j != i;
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
          const int slot = n + __popc(m & ((1u << lane) - 1u));
          if (slot < maxneigh) list[(size_t) slot * stride + i] = j;
        }
        n += __popc(m);
      }
    }
  }
  if (lane == 0) {
    num[i] = n;
    if (n > maxneigh) atomicMax(overflow, n);
  }
}

__global__ void __launch_bounds__(128)
k_elem_list(const double *__restrict__ ex, const int *__restrict__ bin,
            const int *__restrict__ bstart, const int *__restrict__ bmem,
            const double4 *__restrict__ bx, const int *__restrict__ stencil, int nstencil,
            int mbins, int nlocal, double cutsq, int maxneigh, int stride,
            int *__restrict__ num, int *__restrict__ list, int *__restrict__ overflow) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nlocal) return;
  const double xt = ex[3 * i], yt = ex[3 * i + 1], zt = ex[3 * i + 2];
  const int ib = bin[i];
  int n = 0;
  for (int k = 0; k < nstencil; k++) {
    int b = ib + __ldg(stencil + k);
    if (b < 0 || b >= mbins) continue;
    int p1 = __ldg(bstart + b + 1);
    for (int p = __ldg(bstart + b); p < p1; p++) {
      int j = __ldg(bmem + p);
      if (j == i) continue;
      double4 xj = bx[p];
      double dx = xt - xj.x, dy = yt - xj.y, dz = zt - xj.z;
      double rsq = dx * dx + dy * dy + dz * dz;
      if (rsq <= cutsq) {
        if (n < maxneigh) list[(size_t) n * stride + i] = j;
        n++;
      }
    }
  }
  num[i] = n;
  if (n > maxneigh) atomicMax(overflow, n);
}

__global__ void k_split_hi(const double4 *__restrict__ x, float4 *__restrict__ xh, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 p = x[i];
  xh[i] = make_float4((float) p.x, (float) p.y, (float) p.z, 0.f);
}

// the ghosts' positions (ghosts.cuh) with the float copies of all atoms
__global__ void k_forward_split(double4 *__restrict__ x, const int *__restrict__ send, int nlocal,
                                int nall, SwapChain c, float4 *__restrict__ xh) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nall) return;
  double4 p;
  if (i >= nlocal) {
    p = ghost_position(x, c, send, nlocal, i);
    x[i] = p;
  } else {
    p = x[i];
  }
  xh[i] = make_float4((float) p.x, (float) p.y, (float) p.z, 0.f);
}

// Sub-element centres (full_node_neighbor.cpp:137-143)
__global__ void k_sub_centres(const double *__restrict__ nodex, int nelem, ElemTables t,
                              double4 *__restrict__ subc) {
  int tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= nelem * t.nsub) return;
  int e = tid / t.nsub, isub = tid % t.nsub;
  const double *C = t.spa_center_sub + (size_t) isub * NPE;
  const double *nx = nodex + 24 * (size_t) e;
  double a = 0.0, b = 0.0, c = 0.0;
#pragma unroll
  for (int k = 0; k < NPE; k++) {
    a += C[k] * nx[3 * k];
    b += C[k] * nx[3 * k + 1];
    c += C[k] * nx[3 * k + 2];
  }
  subc[tid] = make_double4(a, b, c, 0.0);
}

// Integration-point lists, one warp per row.  Sites are tested in FP32 on
// coordinates relative to node 0 of the row's element, interpolated from float
// nodes and weights: with R the largest such coordinate a difference is within
// 22 u R (u = 2^-24), and FP64 arithmetic on absolute coordinates up to X
// places the pair within 24 * 2^-53 X of that.  Only a distance that these
// bounds leave open (near the cutoff, or near the 1e-2 that excludes the row's
// own site) is formed in FP64, as the reference does (Interpolate_to_atom_vec,
// element.cpp:1226-1272, then full_node_neighbor.cpp:150-190).  The FP64
// positions of all sites, local and ghost, took 579 us and the FP64 tests
// 636 us for 1,024 elements of 1,331 sites.
__device__ __forceinline__ double node_interp(const double *__restrict__ N,
                                              const double *__restrict__ x, int d) {
  double a = 0;
#pragma unroll
  for (int k = 0; k < NPE; k++) a += N[k] * x[3 * k + d];
  return a;
}

__global__ void __launch_bounds__(128)
k_ip_list(const double *__restrict__ nodex, const double *__restrict__ ex,
          const int *__restrict__ etype, const int *__restrict__ row_elem,
          const int *__restrict__ row_jj, int nrows, const int *__restrict__ enum_,
          const int *__restrict__ elist, int estride, const double4 *__restrict__ subc,
          const float4 *__restrict__ spa_inter_f, const int *__restrict__ site_base, ElemTables t,
          double cut_elesq, double cut_subelesq, double cutsq, int maxip, int rowstride,
          int *__restrict__ ipnum, int *__restrict__ ipent, int *__restrict__ overflow) {
  __shared__ float s_nodes[4][24];
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= nrows) return;
  float *s_x = s_nodes[threadIdx.x >> 5];
  const unsigned lt_mask = (1u << lane) - 1u;
  const int e = row_elem[r], jj = row_jj[r], ty = etype[e];
  const double *N = t.spa_int + ((size_t) t.int_off[ty] + jj) * NPE;
  const double *nxe = nodex + 24 * (size_t) e;
  // the row's point: lanes 0..2 a component each
  const double pd = lane < 3 ? node_interp(N, nxe, lane) : 0.0;
  const double ix = __shfl_sync(0xffffffffu, pd, 0), iy = __shfl_sync(0xffffffffu, pd, 1),
               iz = __shfl_sync(0xffffffffu, pd, 2);
  const double x0 = nxe[lane % 3];  // node 0, this lane's component
  const float pf = lane < 3 ? (float) (pd - x0) : 0.f;
  const float px = __shfl_sync(0xffffffffu, pf, 0), py = __shfl_sync(0xffffffffu, pf, 1),
              pz = __shfl_sync(0xffffffffu, pf, 2);
  const float rc = sqrtf((float) cutsq);
  int n = 0;
  const int nsub = t.nsub;
  const int ne = enum_[e];
  // neighbor elements first, then the element itself (self: rsq > 1e-4)
  for (int ll = 0; ll <= ne; ll++) {
    const bool self = ll == ne;
    const int j = self ? e : elist[(size_t) ll * estride + e];
    if (!self) {
      const double cx = ex[3 * j], cy = ex[3 * j + 1], cz = ex[3 * j + 2];
      double npdis = (ix - cx) * (ix - cx) + (iy - cy) * (iy - cy) + (iz - cz) * (iz - cz);
      if (!(npdis <= cut_elesq)) continue;
    }
    // the element's nodes relative to node 0 of the row's element
    float R = 0.f, X = 0.f;
    __syncwarp();
    if (lane < 24) {
      const double v = nodex[24 * (size_t) j + lane];
      const float f = (float) (v - x0);
      s_x[lane] = f;
      R = fmaxf(fabsf(f), fabsf(pf));
      X = fabsf((float) v);
    }
    __syncwarp();
    R = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(R)));
    X = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(X)));
    const float delta = 1.7320509f * (24.f * 5.9604645e-8f * R + 32.f * 1.110223e-16f * X);
    const float a0 = rc * 0.999999f - delta, a1 = rc * 1.000001f + delta, a2 = 0.01f * 1.000001f + delta;
    const float lo = a0 > 0.f ? a0 * a0 * 0.99999f : -1.f, hi = a1 * a1 * 1.00001f;
    const float near0 = self ? a2 * a2 * 1.00001f : -1.f;
    // sub-element centre test, lanes over sub-elements
    for (int s0 = 0; s0 < nsub; s0 += 32) {
      int isub = s0 + lane;
      bool pass = false;
      if (isub < nsub) {
        double4 sc = subc[(size_t) j * nsub + isub];
        double nps = (ix - sc.x) * (ix - sc.x) + (iy - sc.y) * (iy - sc.y) +
                     (iz - sc.z) * (iz - sc.z);
        pass = nps <= cut_subelesq;
      }
      unsigned b = __ballot_sync(0xffffffffu, pass);
      // process passing sub-elements of this chunk in order
      while (b) {
        int bit = __ffs(b) - 1;
        b &= b - 1;
        int isub2 = s0 + bit;
        int first = t.sub_first[isub2], cnt = t.sub_first[isub2 + 1] - first;
        const int sb = site_base[j];
        const size_t at0 = (size_t) t.inter_off[etype[j]];
        for (int m0 = 0; m0 < cnt; m0 += 32) {
          int mm = m0 + lane;
          bool hit = false;
          int sid = 0;
          if (mm < cnt) {
            int nj = t.list_inter_sub[first + mm];
            sid = sb + nj;
            const float4 w0 = __ldg(spa_inter_f + 2 * (at0 + nj));
            const float4 w1 = __ldg(spa_inter_f + 2 * (at0 + nj) + 1);
            const float w[NPE] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
            float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
            for (int k = 0; k < NPE; k++) {
              sx = __fmaf_rn(w[k], s_x[3 * k], sx);
              sy = __fmaf_rn(w[k], s_x[3 * k + 1], sy);
              sz = __fmaf_rn(w[k], s_x[3 * k + 2], sz);
            }
            const float gx = sx - px, gy = sy - py, gz = sz - pz;
            const float g = gx * gx + gy * gy + gz * gz;
            hit = g < lo && g > near0;
            if (!hit && !(g > hi)) {
              const double *S = t.spa_inter + (at0 + nj) * NPE;
              const double *xj = nodex + 24 * (size_t) j;
              const double dx = node_interp(S, xj, 0) - ix, dy = node_interp(S, xj, 1) - iy,
                           dz = node_interp(S, xj, 2) - iz;
              const double rsq = dx * dx + dy * dy + dz * dz;
              hit = self ? (rsq <= cutsq && rsq > 1.0e-4) : (rsq <= cutsq);
            }
          }
          unsigned hb = __ballot_sync(0xffffffffu, hit);
          if (hit) {
            int slot = n + __popc(hb & lt_mask);
            if (slot < maxip) ipent[(size_t) slot * rowstride + r] = sid;
          }
          n += __popc(hb);
        }
      }
    }
  }
  if (lane == 0) {
    ipnum[r] = n;
    if (n > maxip) atomicMax(overflow, n);
  }
}

}  // namespace

void launch_atom_list(const double4 *x, const int *bin, const int *bstart, const float4 *bxf,
                      const int2 *runs, int nruns, int mbins, int nlocal, double cutsq, float lo,
                      float hi, int maxneigh, int stride, int *num, int *list, int *overflow,
                      cudaStream_t s) {
  if (nlocal <= 0) return;
  k_atom_list<<<nblk((long long) nlocal * 32, AL_BLOCK), AL_BLOCK, 0, s>>>(
      x, bin, bstart, bxf, runs, nruns, mbins, nlocal, cutsq, lo, hi, maxneigh, stride, num, list,
      overflow);
  check(cudaGetLastError(), "atom_list");
}

void launch_elem_list(const double *ex, const int *bin, const int *bstart, const int *bmem,
                      const double4 *bx, const int *stencil, int nstencil, int mbins,
                      int nlocal, double cutsq, int maxneigh, int stride, int *num, int *list,
                      int *overflow, cudaStream_t s) {
  if (nlocal <= 0) return;
  k_elem_list<<<nblk(nlocal, 128), 128, 0, s>>>(ex, bin, bstart, bmem, bx, stencil, nstencil,
                                                 mbins, nlocal, cutsq, maxneigh, stride, num,
                                                 list, overflow);
  check(cudaGetLastError(), "elem_list");
}

void launch_split_hi(const double4 *x, float4 *xh, int n, cudaStream_t s) {
  if (n <= 0) return;
  k_split_hi<<<nblk(n, 256), 256, 0, s>>>(x, xh, n);
  check(cudaGetLastError(), "split_hi");
}

void launch_forward_split(double4 *x, const int *send, int nlocal, int nghost, const SwapChain &c,
                          float4 *xh, cudaStream_t s) {
  const int n = nlocal + nghost;
  if (n <= 0) return;
  k_forward_split<<<nblk(n, 256), 256, 0, s>>>(x, send, nlocal, n, c, xh);
  check(cudaGetLastError(), "forward_split");
}

void launch_sub_centres(const double *nodex, int nelem, ElemTables t, double4 *subc,
                        cudaStream_t s) {
  if (nelem <= 0) return;
  k_sub_centres<<<nblk((long long) nelem * t.nsub, 128), 128, 0, s>>>(nodex, nelem, t, subc);
  check(cudaGetLastError(), "sub_centres");
}

void launch_ip_list(const double *nodex, const double *ex, const int *etype,
                    const int *row_elem, const int *row_jj, int nrows, const int *enum_,
                    const int *elist, int estride, const double4 *subc,
                    const float4 *spa_inter_f, const int *site_base, ElemTables t, double cut_elesq, double cut_subelesq,
                    double cutsq, int maxip, int rowstride, int *ipnum, int *ipent,
                    int *overflow, cudaStream_t s) {
  if (nrows <= 0) return;
  k_ip_list<<<nblk((long long) nrows * 32, 128), 128, 0, s>>>(
      nodex, ex, etype, row_elem, row_jj, nrows, enum_, elist, estride, subc, spa_inter_f,
      site_base, t, cut_elesq, cut_subelesq, cutsq, maxip, rowstride, ipnum, ipent, overflow);
  check(cudaGetLastError(), "ip_list");
}

}  // namespace cacg
