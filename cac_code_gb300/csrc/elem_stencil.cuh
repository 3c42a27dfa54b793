// Mixed EAM element passes over a shared stencil: 32 elements a warp, one lane
// each, all walking the same list of sites.  Included by k_mixed.cu (inside its
// namespace).
//
// The element passes of one warp per element (k_elem_rho_fused,
// k_elem_force_fused) spend two thirds of their instructions on what every
// element of a type repeats: decoding the list entries' lattice indices, the
// monomial differences m(p) - m(s) of a row's point p and a site s, and reading
// the coefficient vectors K from shared memory at every entry.  Elements of one
// type in similar shape have the same sites within reach of a row, so the list of
// a row is here one stencil for all elements: its sites' monomials come from
// shared memory, the same for every lane, K lies in each lane's registers, and
// the sums need no shuffles.  The lanes' distances at one entry are nearly the
// same, so a warp's table look-ups fall on a few neighboring lines of the L1 (staged in
// shared memory they take as long, and 96 KB of it keep the atom passes off the SM).
//
// Build: whenever the lists are reordered (k_fused_reorder).  The range of every
// coefficient over all elements bounds each site's distance from below; the sites
// that may lie within r_c + CULL_DELTA of the row in some element are the stencil
// (in site order, at most STENCIL_CAP a row).  k_stencil_check then evaluates them
// for every element: the stencil stands for the lists (state[0]) if the count
// within r_c + CULL_DELTA equals the list's own in every row, so that no pair is
// missing or extra while the lists' culling is good, and if the elements are alike
// enough (at most 1.5 times a mean list within r_c + CULL_D1).  It also keeps each
// entry's least distance: a pass leaves out the entries that no displacement since
// the reorder can have brought within the cutoff.  Otherwise the passes run one
// warp per element from the lists, in the blocks of this launch (elements not alike,
// densities and forces without a stencil / now: 3,664 37 + 71 / 27 + 67 us, 14,400 52 +
// 113 / 40 + 99).
//
// Sums: FP32 over the entries of 8 consecutive stencil places, then double-single,
// whatever was left out, so that leaving entries out changes no bit.
constexpr int STENCIL_TEAM = 256;   // 8 warps: 32 elements, a row a warp at a time
constexpr int STENCIL_TEAMS = 3;    // teams of a block, at most

enum { ST_VALID, ST_BUILT, ST_CHECKED, ST_BAD, ST_SUM, ST_RANGE = 6 };

__device__ __forceinline__ int ordered_int(float v) {
  const int i = __float_as_int(v);
  return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float ordered_float(int i) {
  return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF);
}

struct Monomials {
  float a, b, c, ab, ac, bc, abc;
};

// m(p) - m(s) of a row's point (its lattice indices and fractions) and a site
__device__ __forceinline__ Monomials monomials(const int4 &p, const FusedLat &g, int i, int j, int k) {
  const float ap = (float) p.x * g.ia, bp = (float) p.y * g.ib, cp = (float) p.z * g.ic;
  const float abp = ap * bp;
  Monomials m;
  m.a = (float) (p.x - i) * g.ia;
  m.b = (float) (p.y - j) * g.ib;
  m.c = (float) (p.z - k) * g.ic;
  m.ab = fmaf(ap, m.b, fmaf(bp, m.a, -m.a * m.b));
  m.ac = fmaf(ap, m.c, fmaf(cp, m.a, -m.a * m.c));
  m.bc = fmaf(bp, m.c, fmaf(cp, m.b, -m.b * m.c));
  m.abc = fmaf(abp, m.c, fmaf(cp, m.ab, -m.ab * m.c));
  return m;
}

// The stencil from the coefficients' ranges, by the last block of the reorder to
// finish (one warp a slot).
__device__ void stencil_build(const Stencil &st, const FusedLat &g, const int4 *intp, float4 lim,
                              float *s_lo, float *s_hi) {
  for (int q = threadIdx.x; q < 21; q += blockDim.x) {
    s_hi[q] = ordered_float(__ldcg(st.state + ST_RANGE + q));
    s_lo[q] = -ordered_float(__ldcg(st.state + ST_RANGE + 21 + q));
  }
  __syncthreads();
  for (int q = threadIdx.x; q < 42; q += blockDim.x) st.state[ST_RANGE + q] = (int) 0x80808080;
  if (threadIdx.x < ST_RANGE) st.state[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, per = g.nay * g.naz;
  for (int q = threadIdx.x >> 5; q < st.ns; q += blockDim.x >> 5) {
    const int4 p = intp[st.rows[q]];
    int n = 0;
    for (int s0 = 0; s0 < st.nsites; s0 += 32) {
      const int s = s0 + lane, i = s / per, j = s % per / g.naz, k = s % g.naz;
      const Monomials m = monomials(p, g, i, j, k);
      const float M[7] = {m.a, m.b, m.c, m.ab, m.ac, m.bc, m.abc};
      float near = 0.f;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        float lo = 0.f, hi = 0.f;
#pragma unroll
        for (int c = 0; c < 7; c++) {
          lo += M[c] * (M[c] >= 0.f ? s_lo : s_hi)[3 * c + d];
          hi += M[c] * (M[c] >= 0.f ? s_hi : s_lo)[3 * c + d];
        }
        const float v = fmaxf(fmaxf(lo, -hi) - 1.0e-3f, 0.f);
        near = fmaf(v, v, near);
      }
      // (a row's own site is in no list)
      const bool keep = s < st.nsites && (i != p.x || j != p.y || k != p.z) && near <= lim.w;
      const unsigned b = __ballot_sync(0xffffffffu, keep);
      const int at = n + __popc(b & ((1u << lane) - 1u));
      if (keep && at < STENCIL_CAP) {
        const size_t o = (size_t) q * STENCIL_CAP + at;
        st.mono[2 * o] = make_float4(m.a, m.b, m.c, m.ab);
        st.mono[2 * o + 1] = make_float4(m.ac, m.bc, m.abc, __int_as_float(s));
        st.minsq[o] = 0x7F800000u;
      }
      n += __popc(b);
    }
    if (lane == 0) {
      st.num[q] = min(n, STENCIL_CAP);
      if (n > STENCIL_CAP) st.state[ST_BAD] = 1;
    }
  }
}

// After a reorder: does the stencil stand for every element's lists?  A block takes 32
// elements, a lane each, a warp a slot at a time; the distances as k_fused_reorder forms
// them.  The entries come 32 at a time through shared memory: read one after another from
// memory by one warp for all slots (which a chain of 2,000 and more loads is) the check
// took 556 us for 3,664 elements alike, and 2,030 us for elements that are not (whole
// reorders: 652 -> 152 and 1,960 -> 154 us; 64,000 elements 3,250 -> 1,072 and 10,000 ->
// 1,125).  One element that the stencil does not stand for ends it for all blocks.
constexpr int CHECK_NT = 256;

__global__ void __launch_bounds__(CHECK_NT)
k_stencil_check(Stencil st, const float2 *__restrict__ node_hl, const int *__restrict__ row_first,
                const int4 *__restrict__ nnear_row, int nlocal_e, float4 lim,
                const unsigned *__restrict__ eflags) {
  if (eflags[1] == 0u) return;
  __shared__ float2 s_nx[32 * 25];
  __shared__ float s_k[21][32];
  __shared__ float4 s_ent[CHECK_NT / 32][32][2];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned long long sum = 0;
  for (int e0 = 32 * (int) blockIdx.x; e0 < nlocal_e; e0 += 32 * (int) gridDim.x) {
    if (__syncthreads_or(*(volatile int *) (st.state + ST_BAD))) break;
    const bool live = e0 + lane < nlocal_e;
    for (int i = threadIdx.x; i < 24 * 32; i += CHECK_NT)
      s_nx[i / 24 * 25 + i % 24] = node_hl[24 * (size_t) min(e0 + i / 24, nlocal_e - 1) + i % 24];
    __syncthreads();
    for (int q = w; q < 21; q += CHECK_NT / 32) {
      const ds v = signed_node_sum(s_nx + 25 * lane + q % 3, 3,
                                   (unsigned) (COEF_POS >> (8 * (q / 3 + 1))) & 0xFFu,
                                   (unsigned) (COEF_NEG >> (8 * (q / 3 + 1))) & 0xFFu);
      s_k[q][lane] = v.h + v.l;
    }
    __syncthreads();
    float k[21];
#pragma unroll
    for (int q = 0; q < 21; q++) k[q] = s_k[q][lane];
    const int rf = row_first[live ? e0 + lane : nlocal_e - 1];
    bool bad = false;
    for (int q = w; q < st.ns; q += CHECK_NT / 32) {
      const int n = st.num[q];
      int cnt = 0;
      for (int t0 = 0; t0 < n; t0 += 32) {
        const size_t o = (size_t) q * STENCIL_CAP + t0 + lane;
        __syncwarp();
        if (t0 + lane < n) {
          s_ent[w][lane][0] = __ldcg(st.mono + 2 * o);
          s_ent[w][lane][1] = __ldcg(st.mono + 2 * o + 1);
        }
        __syncwarp();
        unsigned least = 0x7F800000u;  // of this lane's entry
        for (int t = 0; t < min(32, n - t0); t++) {
          const float4 ma = s_ent[w][t][0], mb = s_ent[w][t][1];
          float r = 0.f;
#pragma unroll
          for (int d = 0; d < 3; d++) {
            float v = k[d] * ma.x;
            v = fmaf(k[3 + d], ma.y, v);
            v = fmaf(k[6 + d], ma.z, v);
            v = fmaf(k[9 + d], ma.w, v);
            v = fmaf(k[12 + d], mb.x, v);
            v = fmaf(k[15 + d], mb.y, v);
            v = fmaf(k[18 + d], mb.z, v);
            r = fmaf(v, v, r);
          }
          cnt += r <= lim.w;
          const unsigned u = __reduce_min_sync(0xffffffffu, __float_as_uint(r));
          if (lane == t) least = u;
        }
        if (t0 + lane < n && least < __ldcg(st.minsq + o)) atomicMin(st.minsq + o, least);
      }
      const int4 nn = nnear_row[rf + st.rows[q]];
      bad |= nn.z != cnt;
      if (live) sum += nn.x;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) st.state[ST_BAD] = 1;
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) atomicAdd(reinterpret_cast<unsigned long long *>(st.state + ST_SUM), sum);
  __shared__ int s_last, s_near;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(st.state + ST_CHECKED, 1) == (int) gridDim.x - 1;
    s_near = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  int near = 0;
  for (int q = 0; q < st.ns; q++)
    for (int t = threadIdx.x; t < st.num[q]; t += blockDim.x)
      near += __uint_as_float(__ldcg(st.minsq + (size_t) q * STENCIL_CAP + t)) <= lim.y;
  atomicAdd(&s_near, near);
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long total = *reinterpret_cast<volatile unsigned long long *>(st.state + ST_SUM);
    const int wrong = *reinterpret_cast<volatile int *>(st.state + ST_BAD);
    st.state[ST_VALID] = !wrong && 2.0 * (double) s_near * nlocal_e <= 3.0 * (double) total;
  }
}

// ---- the passes ----

struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 f2_of(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float f2_lo(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return x;
}
__device__ __forceinline__ float f2_hi(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return y;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ void lds_f2x2(unsigned addr, f2 &a, f2 &b) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a.v), "=l"(b.v) : "r"(addr));
}

// knot and fraction of a table argument without conversions: t = 2^23 + floor(p)
// by rounding p + 2^23 down, at most hi = 2^23 + the last knot (also for a NaN);
// the knot m is t's low bits, p - m (at most 1) the fraction.  LOW: p may be below
// 1; the first knot is 1.
template <bool LOW>
__device__ __forceinline__ float knot_of(float p, float hi, int &m) {
  constexpr float TWO23 = 8388608.f;
  float t = __fadd_rd(p, TWO23);
  if (LOW) t = fmaxf(t, TWO23 + 1.f);
  t = fminf(t, hi);
  m = __float_as_int(t) - MAGIC;
  return fminf(p - (t - TWO23), 1.0f);
}
// 1 / sqrt(x), rsqrtf's instruction without its steps for x below 2^-126
__device__ __forceinline__ float rsqrt_normal(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// a team's shared memory, in float2: the coefficients of axes x, y and of z and the
// nodal density ([m][element] each), the nodal densities ([k][element]), the guard
// band's marks, then the elements' nodes (25 to an element: no bank conflicts),
// whose place the rows' forces ([3 j + axis][element]) take afterwards
constexpr int TEAM_KZ = 7 * 32, TEAM_ER = 2 * TEAM_KZ, TEAM_MARK = TEAM_ER + 8 * 32,
              TEAM_NX = TEAM_MARK + 16;
__host__ __device__ constexpr int team_float2(int nf) {
  return TEAM_NX + (nf * 96 > 32 * 25 ? nf * 96 : 32 * 25);
}
constexpr int STENCIL_ENT = 16;  // floats of a staged entry

// The rows' entries, all of them (the choice between stencil and lists does not depend on
// the culling), fit in cap?
__device__ __forceinline__ bool stencil_room(const Stencil &st, const int *slot, int nrow, int cap) {
  int all = 0;
  for (int r = 0; r < nrow; r++) all += st.num[slot[r]];
  return all <= cap;
}

// The stencil's entries in reach (all of them without culling), for the pass's rows,
// into s_ent (every monomial twice: a packed operand for both halves; then whether the
// FP32 sums end here, and the site); s_off[r] the first of row r.
__device__ __forceinline__ void stencil_stage(const Stencil &st, const int *slot, int nrow,
                                              const unsigned *eflags, bool cull, float cutsq,
                                              float *s_ent, int *s_off) {
  const float d = (eflags[1] ? 0.f : 2.0f * sqrtf(__uint_as_float(eflags[0]))) + CULL_MARGIN;
  const float rl = sqrtf(cutsq) + d, lim = cull ? rl * rl * 1.00001f : INFINITY;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int r = w; r < nrow; r += nw) {
    const int q = slot[r], n = st.num[q];
    int c = 0;
    for (int t = lane; t < n; t += 32)
      c += __uint_as_float(st.minsq[(size_t) q * STENCIL_CAP + t]) <= lim;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) s_off[r + 1] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s_off[0] = 0;
    for (int r = 0; r < nrow; r++) s_off[r + 1] += s_off[r];
  }
  __syncthreads();
  for (int r = w; r < nrow; r += nw) {
    const int q = slot[r], n = st.num[q];
    int at = s_off[r];
    for (int t0 = 0; t0 < n; t0 += 32) {
      const int t = t0 + lane;
      const size_t o = (size_t) q * STENCIL_CAP + t;
      const bool in = t < n && __uint_as_float(st.minsq[o]) <= lim;
      const unsigned b = __ballot_sync(0xffffffffu, in);
      if (in) {
        const float4 ma = st.mono[2 * o], mb = st.mono[2 * o + 1];
        // the last entry left of its eight places?
        const bool last = (b & (0xFFu << (lane & 24)) & ~((2u << lane) - 1u)) == 0u;
        float4 *p = reinterpret_cast<float4 *>(s_ent) +
                    (STENCIL_ENT / 4) * (at + __popc(b & ((1u << lane) - 1u)));
        p[0] = make_float4(ma.x, ma.x, ma.y, ma.y);
        p[1] = make_float4(ma.z, ma.z, ma.w, ma.w);
        p[2] = make_float4(mb.x, mb.x, mb.y, mb.y);
        p[3] = make_float4(mb.z, mb.z, last ? 1.f : 0.f, mb.w);
      }
      at += __popc(b);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(STENCIL_TEAM) : "memory");
}

// the elements of [begin, end) that the surrogate leaves: todo[0] of them (zeroed
// before), in any order
__global__ void k_unskipped(const unsigned char *__restrict__ skip, int begin, int end,
                            int *__restrict__ todo) {
  const int lane = threadIdx.x & 31;
  for (int e0 = begin + (int) ((blockIdx.x * blockDim.x + threadIdx.x) & ~31u); e0 < end;
       e0 += gridDim.x * blockDim.x) {
    const int e = e0 + lane;
    const bool left = e < end && !skip[e];
    const unsigned b = __ballot_sync(0xffffffffu, left);
    int at = 0;
    if (lane == 0 && b) at = atomicAdd(todo, __popc(b));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (left) todo[1 + at + __popc(b & ((1u << lane) - 1u))] = e;
  }
}

// DENSITY: EAM nodal densities (rows: the element's 8 nodes) into out = erho; else
// the forces of the rows of nonzero weight gathered onto the nodes, out = nodef.
// Bound by instruction issue (66 to 75 % of the slots).  C5 (499,712 elements):
// densities 550 -> 225 us, forces 1,917 -> 940 us; 64,000 elements: 90 -> 35 and 277 ->
// 138 us.
// LISTED: the listed elements again, any 32 of them a task, with the guard band's pairs
// decided in FP64 and the sums as in the pass itself, so that neither the band's width nor
// a pair that enters it changes a bit beyond the decisions.
template <bool DENSITY, int MODE>
__global__ void __launch_bounds__(STENCIL_TEAM *STENCIL_TEAMS, 1)
k_elem_stencil(FusedArgs a, Stencil st, int cap, const float4 *__restrict__ tab, int nr, float rdr,
               const double *__restrict__ erho, double *__restrict__ out) {
  extern __shared__ float4 smem[];
  __shared__ int s_off[FUSED_MAXF + 1];
  constexpr bool FIX = MODE == LISTED;
  const int nfix = FIX ? min(a.band[0], a.nlocal_e) : 0;
  if (FIX && nfix == 0) return;  // the whole grid (the count is the same for every block)
  const int nrow = DENSITY ? NPE : st.nf;
  float *s_ent = reinterpret_cast<float *>(smem);
  // with a surrogate: the listed elements (k_unskipped), any 32 of them a task
  const int *todo = FIX ? a.band + BAND_LIST : !DENSITY && a.skip ? st.todo + 1 : nullptr;
  const int count = FIX ? nfix : todo ? st.todo[0] : a.e_end - a.e_begin;
  const int ntask = (count + 31) / 32, nteam = blockDim.x / STENCIL_TEAM;
  const int *slot = st.slot + (DENSITY ? st.nf : 0);
  if (st.state[ST_VALID] == 0 || !stencil_room(st, slot, nrow, cap)) {
    if (DENSITY)
      elem_rho_body<1, MODE, true>(a, tab, nr, rdr, out);
    else
      elem_force_body<true, 1, MODE, true>(a, tab, nr, rdr, 0.f, 0.f, erho, out);
    return;
  }
  if ((int) blockIdx.x * nteam >= ntask) {
    if (FIX) band_done(a.band, nfix);
    return;
  }
  stencil_stage(st, slot, nrow, a.eflags, a.nnear_row != nullptr, a.cutsq_f, s_ent, s_off);
  const int team = threadIdx.x / STENCIL_TEAM, tt = threadIdx.x % STENCIL_TEAM;
  const int w = tt >> 5, lane = tt & 31;
  float2 *s_kx = reinterpret_cast<float2 *>(s_ent + (size_t) STENCIL_ENT * cap) +
                 (size_t) team * team_float2(DENSITY ? 0 : nrow);
  float2 *s_kz = s_kx + TEAM_KZ, *s_er = s_kx + TEAM_ER, *s_nx = s_kx + TEAM_NX;
  float2 *s_f = s_nx;
  int *s_mark = reinterpret_cast<int *>(s_kx + TEAM_MARK);
  const int f0 = a.fjj_off[1], ioff = a.int_off[1];  // (one element type)
  const float band_lo = a.band_lo, band_hi = a.band_hi;
  const float knots = 8388608.f + (float) (nr - 1), fknots = 8388608.f + (float) (a.nrho - 1);
  for (int task = blockIdx.x * nteam + team; task < ntask; task += gridDim.x * nteam) {
    const int t0 = 32 * task, ne = min(32, count - t0);
    auto element = [&](int k) { return todo ? todo[t0 + k] : a.e_begin + t0 + k; };
    for (int i = tt; i < 24 * ne; i += STENCIL_TEAM)
      s_nx[i / 24 * 25 + i % 24] = __ldg(a.node_hl + 24 * (size_t) element(i / 24) + i % 24);
    if (!DENSITY) {
      const int el = tt >> 3;
      const ds v = el < ne ? ds_of_double(__ldg(erho + NPE * (size_t) element(el) + (tt & 7)))
                           : ds{0.f, 0.f};
      s_er[32 * (tt & 7) + el] = make_float2(v.h, v.l);
    }
    if (tt < 32) s_mark[tt] = 0;
    team_sync(team);
    // the coefficients: a warp an axis (3: the nodal densities), a lane an element
    if (w < (DENSITY ? 3 : 4)) {
      auto node = [&](int k) {
        const float2 v = w < 3 ? s_nx[25 * lane + 3 * k + w] : s_er[32 * k + lane];
        return ds{v.x, v.y};
      };
      const ds n0 = node(0), n4 = node(4);
      const ds ka = ds_sub(node(1), n0), kb = ds_sub(node(3), n0), kc = ds_sub(n4, n0);
      const ds x23 = ds_sub(node(2), node(3)), x54 = ds_sub(node(5), n4), x74 = ds_sub(node(7), n4);
      const ds kab = ds_sub(x23, ka), kac = ds_sub(x54, ka), kbc = ds_sub(x74, kb);
      const ds kabc = ds_sub(ds_sub(ds_sub(node(6), node(7)), x54), kab);
      const ds k[7] = {ka, kb, kc, kab, kac, kbc, kabc};
      float *o = reinterpret_cast<float *>(w < 2 ? s_kx : s_kz) + (w & 1);
#pragma unroll
      for (int m = 0; m < 7; m++) o[2 * (32 * m + lane)] = k[m].h + k[m].l;
    } else if (DENSITY && w == 3) {
#pragma unroll
      for (int m = 0; m < 7; m++) s_kz[32 * m + lane].y = 0.f;
    }
    team_sync(team);
    f2 kx[7], kz[7];
#pragma unroll
    for (int m = 0; m < 7; m++) {
      const float2 u = s_kx[32 * m + lane], v = s_kz[32 * m + lane];
      kx[m] = f2_of(u.x, u.y);
      kz[m] = f2_of(v.x, v.y);
    }
    float far = 0.f;  // the largest squared distance up to the guard band's end
    const int mine = FIX ? element(min(lane, ne - 1)) : 0;
    for (int r = w; r < nrow; r += STENCIL_TEAM / 32) {
      const int jj = FIX ? (DENSITY ? a.node_list[NPE + r] : a.fjj[f0 + r]) : 0;
      float fpi = 0.f, rho_p = 0.f;
      if (!DENSITY)
        fpi = row_fprime_ds<32>(a.spa_int_hl + ((size_t) ioff + a.fjj[f0 + r]) * NPE, s_er + lane,
                                a.frho_ds, a.nrho, a.rdrho_ds, rho_p);
      dsacc fx, fy, fz;
      float px = 0.f, py = 0.f, pz = 0.f;
      unsigned at = (unsigned) __cvta_generic_to_shared(s_ent) + 4 * STENCIL_ENT * s_off[r];
      const unsigned end = (unsigned) __cvta_generic_to_shared(s_ent) + 4 * STENCIL_ENT * s_off[r + 1];
#pragma unroll 1
      for (; at < end; at += 4 * STENCIL_ENT) {
        f2 m0, m1, m2, m3, m4, m5, m6, fl;
        lds_f2x2(at, m0, m1);
        lds_f2x2(at + 16, m2, m3);
        lds_f2x2(at + 32, m4, m5);
        lds_f2x2(at + 48, m6, fl);
        f2 u = f2_mul(kx[0], m0), v = f2_mul(kz[0], m0);
        u = f2_fma(kx[1], m1, u);
        v = f2_fma(kz[1], m1, v);
        u = f2_fma(kx[2], m2, u);
        v = f2_fma(kz[2], m2, v);
        u = f2_fma(kx[3], m3, u);
        v = f2_fma(kz[3], m3, v);
        u = f2_fma(kx[4], m4, u);
        v = f2_fma(kz[4], m4, v);
        u = f2_fma(kx[5], m5, u);
        v = f2_fma(kz[5], m5, v);
        u = f2_fma(kx[6], m6, u);
        v = f2_fma(kz[6], m6, v);
        const float dx = f2_lo(u), dy = f2_hi(u), dz = f2_lo(v);
        const float rsq = fmaf(dz, dz, fmaf(dx, dx, dy * dy));
        bool in = rsq <= band_hi;
        if (FIX)
          in = stencil_band64(in && rsq >= band_lo && lane < ne, rsq < a.cutsq_f,
                              a.spa_int + ((size_t) ioff + jj) * NPE,
                              a.spa_inter + ((size_t) a.inter_off[1] + __float_as_int(f2_hi(fl))) * NPE,
                              a.nodex, mine, a.cutsq);
        if (in) {
          if (!FIX) far = fmaxf(far, rsq);
          const float recip = rsqrt_normal(rsq);
          int m;
          const float p = knot_of<false>(fmaf(rsq * recip, rdr, 1.0f), knots, m);
          const float4 t0 = __ldg(tab + (DENSITY ? m : FTAB_W * m));
          if (DENSITY) {
            px += ((t0.x * p + t0.y) * p + t0.z) * p + t0.w;
          } else {
            // F' of the site at rho(p) - sum Rm (m(p) - m(s)), as fprime32
            int h;
            const float q = knot_of<true>(fmaf(rho_p - f2_hi(v), a.rdrho, 1.0f), fknots, h);
            const float4 c = __ldg(a.fp4 + h), t1 = __ldg(tab + FTAB_W * m + 1);
            const float fpj = (c.x * q + c.y) * q + c.z;
            // force_spline
            const float rhoip = (t0.x * p + t0.y) * p + t0.z;
            const float z2 = ((t0.w * p + t1.x) * p + t1.y) * p + t1.z;
            const float z2p = ((3.0f * t0.w * p + 2.0f * t1.x) * p + t1.y) * rdr;
            const float phi = z2 * recip;
            const float phip = z2p * recip - phi * recip;
            const float psip = (fpi + fpj) * rhoip + phip;
            const float fpair = -psip * recip;
            px += dx * fpair;
            py += dy * fpair;
            pz += dz * fpair;
          }
        }
        if (f2_lo(fl) != 0.f) {
          fx.add(px);
          if (!DENSITY) {
            fy.add(py);
            fz.add(pz);
          }
          px = py = pz = 0.f;
        }
      }
      if (DENSITY) {
        if (lane < ne) out[NPE * (size_t) element(lane) + r] = fx.value();
      } else {
        s_f[32 * (3 * r) + lane] = make_float2(fx.h, fx.l);
        s_f[32 * (3 * r + 1) + lane] = make_float2(fy.h, fy.l);
        s_f[32 * (3 * r + 2) + lane] = make_float2(fz.h, fz.l);
      }
    }
    // an element with a pair in the guard band is run again
    if (!FIX && far >= band_lo && lane < ne) s_mark[lane] = 1;
    team_sync(team);
    if (!DENSITY)
      for (int i = tt; i < 24 * ne; i += STENCIL_TEAM) {  // the nodal gather, rows ascending
        const int el = i / 24, q = i % 24 / 3, c = i % 3;
        const float *wt = a.wnf + (size_t) f0 * NPE + q;
        dsacc acc;
        for (int j = 0; j < nrow; j++) {
          const float wq = __ldg(wt + j * NPE);
          const float2 f = s_f[32 * (3 * j + c) + el];
          acc.add(__fmul_rn(wq, f.x));
          acc.add(__fmul_rn(wq, f.y));
        }
        out[24 * (size_t) element(el) + i % 24] = acc.value();
      }
    if (!FIX && tt < ne && s_mark[tt]) band_list(a.band, element(tt), a.nlocal_e);
    team_sync(team);
  }
  if (FIX) band_done(a.band, nfix);
}
