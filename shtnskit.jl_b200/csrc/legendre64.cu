// legendre64.cu — FP64 associated-Legendre contraction kernels on the FP64 tensor cores
// (three or more fields; simt.cu takes one and two).
//
// Both directions work per order m on latitude PAIRS (i, nlat-1-i) folded by
// equatorial symmetry: P_l^m(-x) = (-1)^(l-m) P_l^m(x), so every contraction is
// split into degrees of even (E) and odd (O) parity l-m:
//   synthesis  W[pair, col] = sum_l P_l(x_pair) a[l, col]
//   analysis   a[l, col]    = sum_pair P_l(x_pair) W[pair, col]
// with col = (field, re|im), on mma.sync m16n8k4 .f64 (512 FMAs in 32 cycles of an SM
// sub-partition, the FP64 units' full rate).
//
// P is regenerated where it is used: the c-scaled recurrence
//   r_l = alpha_l x r_{l-1} - r_{l-2},   P_l^m = c_l r_l
// (one DMUL + one DFMA per value) runs in the lanes whose MMA fragment needs the value, so it
// passes through neither global nor shared memory. Each lane's chain starts from the plan's
// recurrence checkpoints (every ckstep degrees), which carry the reference's extended-range
// sectoral seed (values below 2^-480 are zero before the pair's start degree).
#include <climits>

#include "kernels.cuh"

namespace shtb {

__device__ __forceinline__ double factor_at(const PlanDev& P, const Factors& F, long long poff, int l, int m) {
  double s = (m == 0) ? F.mf0 : F.mf1;
  if (F.fac) s *= F.fac[poff + (l - m)];
  if (F.sc_mode) {
    const double q = F.sc[l + (long long)(P.lmax + 1) * m];
    s = (F.sc_mode == 1) ? s * q : s / q;
  }
  return s;
}

// D (16x8) += A (16x4, row-major) B (4x8, column-major), FP64. Fragments per lane
// (g = lane / 4, t = lane % 4): a0 = A[g][t], a1 = A[g + 8][t]; b0 = B[t][g];
// d0, d1 = D[g][2t], D[g][2t + 1]; d2, d3 = D[g + 8][2t], D[g + 8][2t + 1].
__device__ __forceinline__ void dmma_16x8x4(double (&d)[4], double a0, double a1, double b0) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ void cp16(void* smem, const void* gmem, unsigned src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp8(void* smem, const void* gmem, unsigned src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp4(void* smem, const void* gmem, unsigned src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------------------
// synthesis: CTA = (64 MT pairs, order m, 4 NT fields), four warps of 16 MT pairs
// ---------------------------------------------------------------------------
// P never leaves the registers. In the A fragment lane (g, t) holds rows g and g + 8 of
// column t; with rows = latitude pairs, that lane runs the recurrence of its own pairs over
// the t-th quarter of the order's degrees, so at step s the four columns are degrees
// lbeg + t Q + s (Q even: one parity) and every lane's new P value is the A operand as it
// comes. The contraction over degrees sums in the accumulators of the step's parity whatever
// the order, so nothing is exchanged between lanes. The coefficients of the four degrees (B
// fragment: column g, degree t) come from shared memory, kSynSteps steps per stage, filled by
// cp.async two stages ahead; the skew 4 t doubles and the row stride = 2 mod 16 doubles keep
// both the 16-byte writes and the fragment reads free of bank conflicts. Per step a warp
// issues MT NT MMAs (512 FMAs each) for 3 FP64 operations per P value, 2 MT values a lane.
constexpr int kSynSteps = 8;
constexpr int kSynStages = 3;
constexpr int kSynThreads = 128;

template <int NT>
struct SynSmem {
  static constexpr int NF = 4 * NT;                          // fields per CTA
  static constexpr int RS = 8 * NT + 2;                      // doubles per degree
  static constexpr int STAGE = 4 * kSynSteps * RS + 16;      // doubles
  static constexpr int TAB = kSynStages * STAGE;             // then alpha and the factor of every degree
  static constexpr int kPad = 8;                             // steps past lend of the last quarter
  static size_t bytes(int ndeg) { return (size_t)(TAB + 2 * (ndeg + kPad)) * 8; }
};

template <int NT, int MT>
__global__ void __launch_bounds__(kSynThreads, NT == 4 ? 4 : 1)
    leg_syn64_kernel(PlanDev P, CoefSrc src, Factors F, double2* __restrict__ W, int nf, int row_end) {
  using SM = SynSmem<NT>;
  constexpr int NF = SM::NF, RS = SM::RS, KS = kSynSteps;
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_lmin;
  __shared__ double2 s_start[64 * MT];   // start states of the CTA's pairs
  const int im = blockIdx.y, m = im * P.mres;
  const int kb = blockIdx.z * NF;
  const int npair = P.npair;
  const long long poff = P.off[im];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int row0 = (blockIdx.x * 4 + warp) * 16 * MT + g;    // pairs row0 + 16 i + 8 h
  const int lend = min(row_end, P.lrec), ndeg = lend - m + 1;
  double* sAl = sm + SM::TAB;
  double* sFa = sAl + ndeg + SM::kPad;
  if (tid == 0) s_lmin = INT_MAX;
  // everything the first degrees need that does not depend on where they start
  double x[MT][2], ra[MT][2], rb[MT][2];
  int l0[MT][2];
  int mn = INT_MAX / 2;
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int p = row0 + 16 * i + 8 * h;
      l0[i][h] = p < npair ? P.l0[(size_t)im * npair + p] : INT_MAX / 2;
      x[i][h] = p < npair ? P.x[p] : 0.0;
      ra[i][h] = rb[i][h] = 0.0;
      mn = min(mn, l0[i][h]);
    }
  for (int i = tid; i < 64 * MT; i += kSynThreads) {
    const int p = blockIdx.x * (64 * MT) + i;
    s_start[i] = p < npair ? P.start[(size_t)im * npair + p] : make_double2(0.0, 0.0);
  }
#pragma unroll 4
  for (int i = tid; i < ndeg + SM::kPad; i += kSynThreads) {
    const bool in = i < ndeg;
    sAl[i] = in ? P.alpha[poff + i] : 0.0;
    sFa[i] = in ? factor_at(P, F, poff, m + i, m) : 0.0;
  }
  __syncthreads();
  mn = __reduce_min_sync(0xffffffffu, mn);
  if (lane == 0) atomicMin(&s_lmin, mn);
  __syncthreads();
  // degrees from lbeg (an even distance from m, no pair starts below it), a quarter per t
  const int lbeg = m + ((max(s_lmin, m) - m) & ~1);
  const int nd = lend - lbeg + 1;                            // <= 0: no pair starts in range
  const int Q = nd > 0 ? ((nd + 3) / 4 + 1) & ~1 : 0;
  const int nch = (Q + KS - 1) / KS;
  const int lq = lbeg + t * Q;                               // this lane's first degree
  const long long cbase = src.packed == 1 ? (poff - m)
                          : src.packed == 2 ? lm_base(P.lmax, P.mres, m) : (long long)m * src.ld_m;
  const double2* st0 = s_start + warp * 16 * MT + g;

  auto stage = [&](int c, int slot) {
    double* B = sm + slot * SM::STAGE;
    for (int idx = tid; idx < NF * 4 * KS; idx += kSynThreads) {
      const int s = idx % KS, q = (idx / KS) & 3, fl = idx / (4 * KS);
      const int l = lbeg + q * Q + c * KS + s, kf = kb + fl;
      const bool ok = c * KS + s < Q && l <= lend && kf < nf;
      const double2* gp = ok ? src.ptr + (long long)kf * src.ld_k + cbase + l : src.ptr;
      cp16(B + (q * KS + s) * RS + 4 * q + 2 * fl, gp, ok ? 16u : 0u);
    }
  };
  for (int c = 0; c < 2; ++c) {
    if (c < nch) stage(c, c);
    cp_commit();
  }
  // state before degree lq: the checkpoint at or below it, rolled forward
  {
    const int cs = P.ckstep;
    const bool in = nd > 0 && lq <= lend;
    const int ks = in ? (lq - m) / cs : 0, lk = m + ks * cs, nroll = in ? lq - lk : 0;
    const int mroll = __reduce_max_sync(0xffffffffu, nroll);
    const double2* ck = P.ckpt + (size_t)(P.ckbase[im] + ks) * npair + row0;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (in && row0 + 16 * i + 8 * h < npair) {
          const double2 v = ck[16 * i + 8 * h];
          ra[i][h] = v.x;
          rb[i][h] = v.y;
        }
    for (int k = 0; k <= mroll; ++k) {
      if (k > nroll || !in) continue;
      const int l = lk + k;
      const double al = sAl[l - m];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (l == l0[i][h]) {
            ra[i][h] = st0[16 * i + 8 * h].x;
            rb[i][h] = st0[16 * i + 8 * h].y;
          }
          if (k == nroll) continue;   // the state before lq, its own start included
          const double r = fma(al * x[i][h], ra[i][h], -rb[i][h]);
          rb[i][h] = ra[i][h];
          ra[i][h] = r;
        }
    }
  }

  double acc[2][MT][NT][4];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][i][j][q] = 0.0;

  int slot = 0;
  for (int c = 0; c < nch; ++c) {
    cp_wait_group<1>();
    __syncthreads();   // stage c is filled; stage c - 1 is read by every warp
    if (c + 2 < nch) stage(c + 2, slot == 0 ? 2 : slot - 1);
    cp_commit();
    const double* B = sm + slot * SM::STAGE + t * (KS * RS + 4) + g;
    slot = slot == 2 ? 0 : slot + 1;
    const int s0 = c * KS, ns = min(KS, Q - s0), ls = lq + s0;
    const double* al = sAl + (ls - m);
    const double* fa = sFa + (ls - m);
    bool some = false, start = false;   // a pair has begun by the chunk's end; one begins inside it
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        some |= l0[i][h] < ls + ns;
        start |= l0[i][h] >= ls + (c == 0) && l0[i][h] < ls + ns;
      }
    if (!__any_sync(0xffffffffu, some && ls <= lend)) continue;
    const bool slow = __any_sync(0xffffffffu, start) || ns < KS;
    // steps past lend (4 Q <= nd + 7) read zeros from the padding
    auto step = [&](int s, int par, double a_l, double f_l, bool sel) {
      double a[MT][2], b[NT];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (sel && ls + s == l0[i][h]) {
            ra[i][h] = st0[16 * i + 8 * h].x;
            rb[i][h] = st0[16 * i + 8 * h].y;
          }
          const double r = fma(a_l * x[i][h], ra[i][h], -rb[i][h]);
          rb[i][h] = ra[i][h];
          ra[i][h] = r;
          a[i][h] = r * f_l;
        }
#pragma unroll
      for (int j = 0; j < NT; ++j) b[j] = B[s * RS + 8 * j];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma_16x8x4(acc[par][i][j], a[i][0], a[i][1], b[j]);
    };
    if (!slow) {
#pragma unroll
      for (int s = 0; s < KS; ++s) step(s, s & 1, al[s], fa[s], false);
    } else {
      for (int s = 0; s < ns; s += 2) {
        step(s, 0, al[s], fa[s], true);
        step(s + 1, 1, al[s + 1], fa[s + 1], true);
      }
    }
  }
  cp_wait_group<0>();   // no copy of this thread is in flight when the CTA exits
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int pr = row0 + 16 * i + 8 * h;
      if (pr >= npair) continue;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int kf = kb + 4 * j + t;
        if (kf >= nf) continue;
        double2* w = W + (((size_t)kf * P.nm + im) * 2) * npair + pr;
#pragma unroll
        for (int p = 0; p < 2; ++p) w[(size_t)p * npair] = make_double2(acc[p][i][j][2 * h], acc[p][i][j][2 * h + 1]);
      }
    }
}

template <int NT, int MT>
static int launch_syn_tile(const shtb_plan* p, const CoefSrc& src, const Factors& F, void* W, int nf, int row_end,
                           int mlim, cudaStream_t st) {
  auto kern = leg_syn64_kernel<NT, MT>;
  // shared memory for the longest order (m = 0)
  const size_t smem = SynSmem<NT>::bytes(std::min(row_end, p->lrec) + 1);
  if (smem > 227 * 1024) return set_error(SHTB_ERR_UNSUPPORTED, "lmax too large for the FP64 synthesis kernel");
  SHTB_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                "synthesis smem attr");
  const dim3 grid((p->npair + 64 * MT - 1) / (64 * MT), mlim / p->mres + 1, (nf + 4 * NT - 1) / (4 * NT));
  prof_begin(st);
  kern<<<grid, kSynThreads, smem, st>>>(p->dev, src, F, (double2*)W, nf, row_end);
  SHTB_LAUNCHED("legendre synthesis kernel");
  return SHTB_OK;
}

int launch_leg_syn64(const shtb_plan* p, const CoefSrc& src, const Factors& F, void* W, int nf, int row_end,
                     int mlim, cudaStream_t st) {
  if (nf <= 2) return launch_simt_syn64(p, src, F, W, nf, row_end, mlim, st);
  // 32 columns a warp leave registers for four CTAs an SM, 64 for three: 2424 against 2536 us at
  // lmax 1023 x 64 fields, 57 against 62 at lmax 255 x 32 fields plus a wind field
  if (nf > 8) return launch_syn_tile<4, 1>(p, src, F, W, nf, row_end, mlim, st);
  // narrower tiles: two row tiles per warp share each B fragment where that still leaves four
  // CTAs for every SM
  const bool two = (long long)((p->npair + 127) / 128) * (mlim / p->mres + 1) >= 4ll * p->nsm;
  if (nf > 4)
    return two ? launch_syn_tile<2, 2>(p, src, F, W, nf, row_end, mlim, st)
               : launch_syn_tile<2, 1>(p, src, F, W, nf, row_end, mlim, st);
  return two ? launch_syn_tile<1, 2>(p, src, F, W, nf, row_end, mlim, st)
             : launch_syn_tile<1, 1>(p, src, F, W, nf, row_end, mlim, st);
}

// ---------------------------------------------------------------------------
// analysis: CTA = 64 degrees of one order, 8 MT CG fields; four warps = CG column groups
// x 4 / CG parts of the latitude sum
// ---------------------------------------------------------------------------
// The transposed product a[l, col]^T = sum_pair W[pair, col] P_l(x_pair): A (16 x 4) holds 8
// fields (rows g real, g + 8 imaginary: one 16-byte load of W gives a lane both) at 4 pairs,
// B (4 x 8) the P values of pair t at the degrees t0 + 8 g + s. Lane (g, t) therefore runs one
// recurrence chain of 8 degrees from the plan's checkpoint at t0 + 8 g, and each new value is
// the B operand of step s as it comes, for MT tiles of 8 fields: no P panel, no shared memory
// and no barrier in the loop. Each step has its own accumulators (8 steps x MT x 4 doubles).
// Four pairs take 8 chain steps (2 FP64 operations a lane) and 8 MT MMAs; the operands of
// the next four (MT x 32 bytes of W, a checkpoint, x) load meanwhile.
// Where the checkpoint table does not fit its budget at 8 degrees, the checkpoints are farther
// apart than these chains, and rolling each chain forward from the checkpoint below it costs
// up to ckstep - 8 steps for the 8 that count (analysis of 64 fields: lmax 1799, ckstep 16, 26.4 ms; lmax
// 2047, ckstep 32, 62.3 ms). So
//   ckstep 16    chains have 16 steps (SL = 16, MT = 1: as many accumulators as SL = 8, MT = 2) and
//                tiles 128 degrees; a pair may start in the middle of a chain. 13.2 ms.
//   ckstep >= 32 (SPARSE) a lane rolls one chain from a checkpoint through all the tile's degrees up
//                to the next one, for one of bg = 4 groups of four pairs, and leaves
//                the states at every 8th degree in the ring slots of the bg steps to come: ckstep - 8
//                roll steps per 32 chain steps of a lane. lmax 2047, 64 fields 22.3 ms, 3 fields 11.1 -> 3.4 ms.
constexpr int kAnaThreads = 128;
constexpr int kAnaSteps = 8;             // degrees per chain; 8 chains per tile
static_assert(8 * kAnaSteps == kAnaTile && 16 * kAnaSteps == kSimtTile, "tile lists of the plan");
constexpr int kAnaRing = 4;              // operand ring: steps of four pairs in flight, plus one

// Loads that stay where they are written, ahead of the step's MMAs.
__device__ __forceinline__ double2 ld_here(const double2* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_here(const double* p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int ld_here(const int* p) {
  int v;
  asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

template <int MT, int CG, int SL, bool SPARSE>
__global__ void __launch_bounds__(kAnaThreads, MT * SL == 16 ? 2 : 3)
    leg_ana64_kernel(PlanDev P, const double2* __restrict__ W, int nf, int row_end, int mlim, CoefSink dst, Factors F,
                     int zero_fill) {
  constexpr int KS = 4 / CG, DEG = 8 * SL;
  static_assert(SL == kAnaSteps || (SL == 2 * kAnaSteps && MT == 1 && !SPARSE), "chains");
  __shared__ __align__(16) unsigned char buf[4 * kAnaRing * ((2 * MT + 1) * 512 + 256)];
  __shared__ double s_fac[DEG];   // factors of the tile's degrees, loaded while the sums run
  __shared__ int sl0[SL > kStartStep ? 4 * kAnaRing * 32 : 1];   // start degrees, long chains only
  static_assert((KS - 1) * CG * kAnaSteps * 4 * 32 * 8 <= sizeof(buf), "partial sums");
  const int2 tile = (SL == kAnaSteps ? P.atiles : P.stiles)[blockIdx.x];
  const int im = tile.x, t0 = tile.y, m = im * P.mres;
  const int lend = min(row_end, P.lrec);
  if (m > mlim || t0 > lend) return;
  const int npair = P.npair;
  const long long poff = P.off[im];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int cg = warp % CG, kw = warp / CG;
  const int kb = blockIdx.y * (8 * MT * CG);            // the CTA's first field
  const int kf0 = kb + 8 * MT * cg + g;                 // this lane's field of tile 0
  const int lg = t0 + SL * g;                           // first degree of this lane's chain
  const int tlast = min(t0 + DEG - 1, lend);
  // this lane's chain: its checkpoint, or (SPARSE) that of the chain it rolls from degree lk for
  // the degrees lr .. lr + seg - 1, for group rg of bg groups of pairs; alpha of its steps
  const int cs = SPARSE ? P.ckstep : SL;
  const int bg = SPARSE ? kAnaRing : 1, rg = g & (bg - 1), seg = min(cs, DEG);
  const int lr = SPARSE ? t0 + seg * (g / bg) : lg;
  const int ks = (min(lr, P.lrec) - m) / cs, lk = lr <= P.lrec ? m + ks * cs : lr;
  const double2* ck = P.ckpt + (size_t)(P.ckbase[im] + ks) * npair;
  const int* pl0 = P.l0 + (size_t)im * npair;
  double al[SL];
#pragma unroll
  for (int s = 0; s < SL; ++s) al[s] = (lg + s <= lend) ? P.alpha[poff + (lg + s - m)] : 0.0;
  const size_t wld = (size_t)P.nm * 2 * npair;

  double acc[SL][MT][4];
#pragma unroll
  for (int s = 0; s < SL; ++s)
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[s][i][q] = 0.0;

  // leading groups of 32 pairs that all start above the tile hold only zeros
  const int nk = (npair + 3) / 4;
  const int k0 = npair <= 32 ? 0 : first_live_pair(pl0, npair, tlast + 1) / 4;
  // operand ring: each lane copies its own operands of the next RG - 1 steps (a checkpoint, x,
  // W of MT fields, E and O) and reads them back itself, so no barrier is needed
  constexpr int RG = kAnaRing, NS = 2 * MT + 1;
  double2* ring = reinterpret_cast<double2*>(buf) + (warp * RG * NS) * 32 + lane;
  double* xring = reinterpret_cast<double*>(buf + 4 * RG * NS * 512) + warp * RG * 32 + lane;
  // fields and chains past the end read valid operands, nothing is stored for them; pairs
  // past the end read zeros
  const double2* Wi[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) Wi[i] = W + (size_t)min(kf0 + 8 * i, nf - 1) * wld + (size_t)im * 2 * npair;
  auto fetch = [&](int k, int st) {
    const int p = 4 * k + t;
    const unsigned n = p < npair ? 16u : 0u;
    const int pc = p < npair ? p : 0;
    double2* r = ring + st * (NS * 32);
    if constexpr (!SPARSE) cp16(r, ck + pc, n);
    cp8(xring + st * 32, P.x + pc, n >> 1);
    if constexpr (SL > kStartStep) cp4(sl0 + (warp * RG + st) * 32 + lane, pl0 + pc, n >> 2);
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      cp16(r + (1 + 2 * i) * 32, Wi[i] + pc, n);
      cp16(r + (2 + 2 * i) * 32, Wi[i] + npair + pc, n);
    }
  };
#pragma unroll
  for (int i = 0; i < RG - 1; ++i) {
    fetch(k0 + kw + i * KS, i);
    cp_commit();
  }
  const int lcap = dst.packed == 1 ? lend : min(lend, P.lmax);
  if (tid < DEG && t0 + tid <= lcap) s_fac[tid] = factor_at(P, F, poff, t0 + tid, m);
  __syncthreads();
  int st = 0;
  // SPARSE: checkpoint, x and start degree of the next chain to roll; zeros past the last pair and degree
  double2 rc = make_double2(0.0, 0.0);
  double rx = 0.0;
  int rl0 = INT_MAX, rp = 0;
  auto roll_fetch = [&](int k) {
    rp = 4 * (k + rg * KS) + t;
    rc = make_double2(0.0, 0.0);
    rx = 0.0;
    rl0 = INT_MAX;
    if (rp < npair && lr <= P.lrec) {
      rc = ld_here(ck + rp);
      rx = ld_here(P.x + rp);
      rl0 = ld_here(pl0 + rp);
    }
  };
  if constexpr (SPARSE) roll_fetch(k0 + kw);   // ckstep >= 8 kAnaRing
  for (int k = k0 + kw; k < nk; k += KS) {
    fetch(k + (RG - 1) * KS, st == 0 ? RG - 1 : st - 1);
    cp_commit();
    if constexpr (SPARSE) {
      if (st == 0) {
        // the states of the next bg steps, into their ring slots
        double2* slot = ring - lane + rg * (NS * 32) + t;
        __syncwarp();   // the slots are read
        for (int l = lk;;) {
          if (l == rl0) rc = P.start[(size_t)im * npair + rp];   // starts lie multiples of 8 degrees from m
          if (l >= lr && lr < t0 + DEG) slot[(l - t0) / SL * 4] = rc;
          if (l + SL >= lr + seg) break;
          double a[SL];
#pragma unroll
          for (int s = 0; s < SL; ++s) a[s] = l + s <= P.lrec ? P.alpha[poff + (l + s - m)] : 0.0;
#pragma unroll
          for (int s = 0; s < SL; ++s) {
            const double q = fma(a[s] * rx, rc.x, -rc.y);
            rc.y = rc.x;
            rc.x = q;
          }
          l += SL;
        }
        __syncwarp();
        roll_fetch(k + bg * KS);
      }
    }
    cp_wait_group<RG - 1>();
    const double2* r = ring + st * (NS * 32);
    const double x = xring[st * 32];
    double ra = r[0].x, rb = r[0].y;
    double2 e[MT], o[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      e[i] = r[(1 + 2 * i) * 32];
      o[i] = r[(2 + 2 * i) * 32];
    }
    const int l0 = SL > kStartStep ? sl0[(warp * RG + st) * 32 + lane] : 0;   // 0 past the last pair
    st = st == RG - 1 ? 0 : st + 1;
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      if (SL > kStartStep && s == kStartStep && l0 == lg + s) {   // the pair starts inside the chain
        const double2 v = P.start[(size_t)im * npair + 4 * k + t];
        ra = v.x;
        rb = v.y;
      }
      const double q = fma(al[s] * x, ra, -rb);
      rb = ra;
      ra = q;
#pragma unroll
      for (int i = 0; i < MT; ++i) dmma_16x8x4(acc[s][i], (s & 1) ? o[i].x : e[i].x, (s & 1) ? o[i].y : e[i].y, q);
    }
  }
  cp_wait_group<0>();   // no copy of this thread is in flight when the CTA exits
  if constexpr (KS > 1) {
    // add the parts of the latitude sum: warps kw > 0 hand theirs over in the ring's memory
    double* part = reinterpret_cast<double*>(buf);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < MT * SL / kAnaSteps; ++c) {   // eight steps of one row tile at a time
      const int i = c % MT, s0 = c / MT * kAnaSteps;
      if (c > 0) __syncthreads();
      if (kw > 0) {
        double* d = part + ((kw - 1) * CG + cg) * kAnaSteps * 4 * 32 + lane;
#pragma unroll
        for (int s = 0; s < kAnaSteps; ++s)
#pragma unroll
          for (int q = 0; q < 4; ++q) d[(s * 4 + q) * 32] = acc[s0 + s][i][q];
      }
      __syncthreads();
      if (kw == 0)
        for (int w = 0; w < KS - 1; ++w) {
          const double* d = part + (w * CG + cg) * kAnaSteps * 4 * 32 + lane;
#pragma unroll
          for (int s = 0; s < kAnaSteps; ++s)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[s0 + s][i][q] += d[(s * 4 + q) * 32];
        }
    }
  }
  if (kw == 0) {
    const long long dbase = dst.packed == 1 ? (poff - m)
                            : dst.packed == 2 ? lm_base(P.lmax, P.mres, m) : (long long)m * dst.ld_m;
    // accumulator columns 2t and 2t + 1 are the chains 2t, 2t + 1
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int s = 0; s < SL; ++s) {
        const int l = t0 + SL * (2 * t + c) + s;
        if (l > lcap) continue;
        const double f = s_fac[l - t0];
#pragma unroll
        for (int i = 0; i < MT; ++i)
          if (kf0 + 8 * i < nf)
            dst.ptr[(long long)(kf0 + 8 * i) * dst.ld_k + dbase + l] = make_double2(acc[s][i][c] * f, acc[s][i][2 + c] * f);
      }
  }
  if (zero_fill && !dst.packed && t0 == m) {
    const int nrow = m + max(P.lmax - lcap, 0);  // rows [0, m) and (lcap, lmax]
    const int nfl = min(8 * MT * CG, nf - kb);
    for (int f = warp; f < nfl; f += 4) {
      double2* col = dst.ptr + (long long)(kb + f) * dst.ld_k + (long long)m * dst.ld_m;
      for (int r = lane; r < nrow; r += 32) col[(r < m) ? r : lcap + 1 + (r - m)] = make_double2(0.0, 0.0);
    }
  }
}

template <int MT, int CG, int SL, bool SPARSE>
static int launch_ana_tile(const shtb_plan* p, const void* W, int nf, int row_end, int mlim, const CoefSink& dst,
                           const Factors& F, int zero_fill, cudaStream_t st) {
  const dim3 grid(SL == kAnaSteps ? p->dev.natiles : p->dev.nstiles, (nf + 8 * MT * CG - 1) / (8 * MT * CG));
  prof_begin(st);
  leg_ana64_kernel<MT, CG, SL, SPARSE>
      <<<grid, kAnaThreads, 0, st>>>(p->dev, (const double2*)W, nf, row_end, mlim, dst, F, zero_fill);
  SHTB_LAUNCHED("legendre analysis kernel");
  return SHTB_OK;
}

template <bool SPARSE>
static int launch_ana_short(const shtb_plan* p, const void* W, int nf, int row_end, int mlim, const CoefSink& dst,
                            const Factors& F, int zero_fill, cudaStream_t st) {
  constexpr int SL = kAnaSteps;
  if (nf > 32) return launch_ana_tile<2, 4, SL, SPARSE>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (nf > 16) return launch_ana_tile<2, 2, SL, SPARSE>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (nf > 8) return launch_ana_tile<2, 1, SL, SPARSE>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  return launch_ana_tile<1, 1, SL, SPARSE>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
}

int launch_leg_ana64(const shtb_plan* p, const void* W, int nf, int row_end, int mlim, const CoefSink& dst,
                     const Factors& F, int zero_fill, cudaStream_t st) {
  if (p->npair > 8192) return set_error(SHTB_ERR_UNSUPPORTED, "nlat too large for the FP64 analysis kernel");
  if (nf <= 2) return launch_simt_ana64(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  // chains as long as the checkpoints are apart, up to 16 degrees; beyond, chains of 8 that roll
  if (p->dev.ckstep == kAnaSteps) return launch_ana_short<false>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (p->dev.ckstep > 2 * kAnaSteps) return launch_ana_short<true>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  constexpr int SL = 2 * kAnaSteps;
  if (nf > 16) return launch_ana_tile<1, 4, SL, false>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (nf > 8) return launch_ana_tile<1, 2, SL, false>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  return launch_ana_tile<1, 1, SL, false>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
}

}  // namespace shtb
