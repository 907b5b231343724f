// legendre64.cu — FP64 associated-Legendre contraction kernels on the FP64 tensor cores.
//
// Both directions work per order m on latitude PAIRS (i, nlat-1-i) folded by
// equatorial symmetry: P_l^m(-x) = (-1)^(l-m) P_l^m(x), so every contraction is
// split into degrees of even (E) and odd (O) parity l-m. Per order and parity each
// direction is a dense GEMM whose P operand is regenerated on the fly:
//   synthesis  W[pair, col] = sum_l P_l(x_pair) a[l, col]     (K = degrees)
//   analysis   a[l, col]    = sum_pair P_l(x_pair) W[pair, col] (K = latitude pairs)
// with col = (field, re|im).
//
// P_l^m is never stored in global memory: four producer warps per CTA regenerate the
// panels of the coming K chunks into a ring of shared-memory stages with the c-scaled
// three-term recurrence
//   r_l = alpha_l x r_{l-1} - r_{l-2},   P_l^m = c_l r_l
// (one DMUL + one DFMA per value), started from per-(m, pair) records that carry the
// reference's extended-range sectoral seed (values below 2^-480 are zero until the
// record's first degree l0) and, inside the degree range, from the plan's recurrence
// checkpoints (every ckstep degrees), so the panel of a chunk is many short independent
// chains rather than one long one; they fill the same stage with the chunk's coefficient
// or Fourier panel by cp.async. Eight consumer warps multiply each stage with FP64 MMAs
// (mma.sync m16n8k4 .f64: 512 FMAs per instruction, the DFMA units' full rate at an
// eighth of the issue slots of DFMA code), operands from shared memory, accumulators in
// registers. Stages are handed over on mbarriers (full: panels written and copies landed;
// empty: every consumer warp done), so the producers run up to a ring's depth ahead and
// their latency-bound recurrence, which shares the FP64 pipe with the MMAs, never holds
// the consumers at a CTA-wide barrier. Every wait is bounded (pipe.cuh).
//
// Per-(l, m) multipliers (c_l, normalization, phi scales) are folded into the P panel
// (synthesis) or applied at the store (analysis). Chunks whose P values are all zero
// (every pair of the chunk still below its record's first degree, near the poles at
// high m) are skipped: adding their zeros changes nothing.
#include <climits>

#include "kernels.cuh"
#include "pipe.cuh"

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
#pragma unroll 4
  for (int i = tid; i < ndeg + SM::kPad; i += kSynThreads) {
    const bool in = i < ndeg;
    sAl[i] = in ? P.alpha[poff + i] : 0.0;
    sFa[i] = in ? factor_at(P, F, poff, m + i, m) : 0.0;
  }
  __syncthreads();
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
  // narrower tiles: two row tiles per warp share each B fragment where that still leaves CTAs
  // for every SM
  const bool two = (long long)((p->npair + 127) / 128) * (mlim / p->mres + 1) >= 592;
  if (nf > 4)
    return two ? launch_syn_tile<2, 2>(p, src, F, W, nf, row_end, mlim, st)
               : launch_syn_tile<2, 1>(p, src, F, W, nf, row_end, mlim, st);
  return two ? launch_syn_tile<1, 2>(p, src, F, W, nf, row_end, mlim, st)
             : launch_syn_tile<1, 1>(p, src, F, W, nf, row_end, mlim, st);
}

constexpr int kConsumerWarps = 8;

// Consumer warp layout shared by both directions: per parity an output tile of 64 rows
// by NCOL columns, split over kConsumerWarps / 2 warps as RG row groups x CG column
// groups; a warp holds MT x NT fragments of 16 x 8.
template <int NCOL>
struct WarpTile {
  static constexpr int WPP = kConsumerWarps / 2;   // warps per parity
  static constexpr int RG = NCOL >= 64 ? 2 : 4, CG = WPP / RG;
  static constexpr int MT = 64 / RG / 16, NT = NCOL / CG / 8;
  static constexpr int NF = NCOL / 2;   // fields per CTA
  static_assert(MT >= 1 && NT >= 1 && RG * CG == WPP, "warp tile");
};

constexpr int kProducerWarps = 4;   // one per SM sub-partition, so the recurrence's FP64 work
                                    // spreads over all four FP64 pipes
constexpr int kLegThreads = 32 * (kConsumerWarps + kProducerWarps);

// ---------------------------------------------------------------------------
// analysis: CTA = (128 degrees of order m, NCOL/2 fields), K chunks of kAnaPairs pairs
// ---------------------------------------------------------------------------
constexpr int kAnaPairs = 16;                    // latitude pairs per chunk
constexpr int kAnaAS = kAnaPairs + 4;            // P panel row stride (doubles), = 4 mod 16
constexpr int kAnaBS = 2 * kAnaPairs + 8;        // Fourier panel field stride (doubles), = 8 mod 16
constexpr int kAnaMaxChunks = 512;               // npair <= 8192
constexpr int kAnaStages = 3;

template <int NCOL>
struct AnaSmem {
  static constexpr int NF = WarpTile<NCOL>::NF;
  static constexpr int ABUF = 2 * 64 * kAnaAS;   // [parity][64 rows][pairs]
  static constexpr int BBUF = 2 * NF * kAnaBS;   // [parity][field][pairs x re|im]
  static constexpr int STAGE = ABUF + BBUF;
  static constexpr int ALPH = kAnaStages * STAGE;          // alpha of the tile's 128 degrees
  static constexpr int BAR = ALPH + kAnaTile;              // then full[S], empty[S], flags, chunk list
  static size_t bytes() { return (size_t)BAR * 8 + 2 * kAnaStages * 8 + 16 + (kAnaMaxChunks + 8) * 4; }
};

template <int NCOL>
__global__ void __launch_bounds__(kLegThreads, 1)
    leg_ana64_kernel(PlanDev P, const double2* __restrict__ W, int nf, int row_end, int mlim, CoefSink dst, Factors F,
                     int zero_fill, int* err) {
  using WT = WarpTile<NCOL>;
  using SM = AnaSmem<NCOL>;
  constexpr int NF = WT::NF, S = kAnaStages;
  extern __shared__ __align__(16) double sm[];
  double* salph = sm + SM::ALPH;
  unsigned long long* full = reinterpret_cast<unsigned long long*>(sm + SM::BAR);
  unsigned long long* empty = full + S;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + S);
  int* slist = reinterpret_cast<int*>(empty + S) + 4;   // nonzero chunks, then their count
  const int4 tile = P.atiles[blockIdx.x];
  const int im = tile.x, t0 = tile.y, ck0 = tile.z, m = im * P.mres;
  const int lend = min(row_end, P.lrec);
  if (m > mlim || t0 > lend) return;
  const int kb = blockIdx.y * NF;
  const int npair = P.npair;
  const long long poff = P.off[im];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool producer = warp >= kConsumerWarps;
  const int tlast = min(t0 + kAnaTile - 1, lend);

  if (tid == 0) {
    for (int q = 0; q < S; ++q) {
      pipe_bar_init(&full[q], 32 * kProducerWarps);
      pipe_bar_init(&empty[q], kConsumerWarps);
    }
    *abort_flag = 0;
    pipe_bar_init_fence();
  }
  for (int i = tid; i < kAnaTile; i += kLegThreads) {
    const int l = t0 + i;
    salph[i] = (l <= lend) ? P.alpha[poff + (l - m)] : 0.0;
  }
  // chunks with a nonzero P value: some pair's first significant degree is <= tlast
  const int nch = (npair + kAnaPairs - 1) / kAnaPairs;
  if (warp == 0) {
    int cnt = 0;
    for (int c0 = 0; c0 < nch; c0 += 32) {
      const int c = c0 + lane;
      bool nz = false;
      if (c < nch) {
        int mn = INT_MAX;
        for (int q = 0; q < kAnaPairs; ++q) {
          const int p = c * kAnaPairs + q;
          if (p < npair) mn = min(mn, P.l0[(size_t)im * npair + p]);
        }
        nz = mn <= tlast;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, nz);
      if (nz) slist[cnt + __popc(bal & ((1u << lane) - 1u))] = c;
      cnt += __popc(bal);
    }
    if (lane == 0) slist[kAnaMaxChunks] = cnt;
  }
  __syncthreads();
  const int nz = slist[kAnaMaxChunks];

  if (producer) {
    // every producer thread takes part in every chunk: thread q = 32 w + lane runs the chain
    // of pair q % 16 over the tile's checkpoint segment q / 16 (ckstep degrees)
    const int ptid = tid - 32 * kConsumerWarps, pq = ptid % kAnaPairs, seg = ptid / kAnaPairs;
    const int cs = P.ckstep, nseg = kAnaTile / cs;
    const bool chain = seg < nseg && t0 + seg * cs <= P.lrec;
    for (int ci = 0; ci < nz; ++ci) {
      const int st = ci % S;
      if (ci >= S && !pipe_wait(&empty[st], ((ci / S) - 1) & 1, abort_flag, err)) break;
      const int c = slist[ci];
      double* A = sm + st * SM::STAGE;
      double* B = A + SM::ABUF;
      for (int idx = ptid; idx < 2 * NF * kAnaPairs; idx += 32 * kProducerWarps) {
        const int q = idx % kAnaPairs, rest = idx / kAnaPairs, fl = rest % NF, pr = rest / NF;
        const int pair = c * kAnaPairs + q, kf = kb + fl;
        const bool ok = pair < npair && kf < nf;
        const double2* gp = ok ? W + (((size_t)kf * P.nm + im) * 2 + pr) * npair + pair : W;
        pipe_cp16(B + (pr * NF + fl) * kAnaBS + 2 * q, gp, ok ? 16u : 0u);
      }
      pipe_arrive_cp_async(&full[st]);
      if (seg < nseg) {
        const int p = c * kAnaPairs + pq;
        double x = 0.0, ra = 0.0, rb = 0.0, r0 = 0.0, r1 = 0.0;
        int l0 = INT_MAX / 2;
        if (p < npair && chain) {
          x = P.x[p];
          const double2 stv = P.ckpt[(size_t)(ck0 + seg) * npair + p];
          ra = stv.x;
          rb = stv.y;
          l0 = P.l0[(size_t)im * npair + p];
          const double2 v = P.start[(size_t)im * npair + p];
          r0 = v.x;
          r1 = v.y;
        }
        const int d0 = seg * cs;
        double* Ar = A + pq;
#pragma unroll 4
        for (int s = 0; s < cs; ++s) {
          const int d = d0 + s, l = t0 + d;
          ra = (l == l0) ? r0 : ra;
          rb = (l == l0) ? r1 : rb;
          const double r = fma(salph[d] * x, ra, -rb);
          rb = ra;
          ra = r;
          Ar[((d & 1) * 64 + (d >> 1)) * kAnaAS] = r;
        }
      }
      pipe_arrive(&full[st]);
    }
    pipe_cp_wait_all();   // no copy of this thread is in flight when the CTA exits
    return;
  }

  const int par = warp / WT::WPP, rg = (warp % WT::WPP) / WT::CG, cg = warp % WT::CG;
  const int rowbase = rg * (64 / WT::RG), colbase = cg * (NCOL / WT::CG);
  const int g = lane >> 2, t = lane & 3;
  double acc[WT::MT][WT::NT][4];
#pragma unroll
  for (int i = 0; i < WT::MT; ++i)
#pragma unroll
    for (int j = 0; j < WT::NT; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;

  // 16-row fragments whose first degree lies past lend hold no output: no MMAs for them
  // (m-tiles are in increasing degree order, so live[0] false means none is live)
  bool live[WT::MT];
#pragma unroll
  for (int i = 0; i < WT::MT; ++i) live[i] = t0 + 2 * (rowbase + i * 16) + par <= lend;

  for (int ci = 0; ci < nz; ++ci) {
    const int st = ci % S;
    if (!pipe_wait(&full[st], (ci / S) & 1, abort_flag, err)) break;
    const double* A = sm + st * SM::STAGE + par * 64 * kAnaAS;
    const double* B = sm + st * SM::STAGE + SM::ABUF + par * NF * kAnaBS;
#pragma unroll
    for (int ks = 0; ks < kAnaPairs / 4 && live[0]; ++ks) {
      double a[WT::MT][2], b[WT::NT];
#pragma unroll
      for (int i = 0; i < WT::MT; ++i) {
        const double* pa = A + (rowbase + i * 16 + g) * kAnaAS + ks * 4 + t;
        a[i][0] = pa[0];
        a[i][1] = pa[8 * kAnaAS];
      }
#pragma unroll
      for (int j = 0; j < WT::NT; ++j) {
        const int col = colbase + j * 8 + g;
        b[j] = B[(col >> 1) * kAnaBS + 2 * (ks * 4 + t) + (col & 1)];
      }
#pragma unroll
      for (int i = 0; i < WT::MT; ++i)
        if (live[i]) {
#pragma unroll
          for (int j = 0; j < WT::NT; ++j) dmma_16x8x4(acc[i][j], a[i][0], a[i][1], b[j]);
        }
    }
    __syncwarp();
    if (lane == 0) pipe_arrive(&empty[st]);
  }
  if (*abort_flag) return;

  const long long dbase = dst.packed == 1 ? (poff - m)
                          : dst.packed == 2 ? lm_base(P.lmax, P.mres, m) : (long long)m * dst.ld_m;
  const int lcap = dst.packed == 1 ? lend : min(lend, P.lmax);
#pragma unroll
  for (int i = 0; i < WT::MT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = rowbase + i * 16 + g + 8 * h;
      const int l = t0 + 2 * row + par;
      if (l > lcap) continue;
      const double s = factor_at(P, F, poff, l, m);
#pragma unroll
      for (int j = 0; j < WT::NT; ++j) {
        const int kf = kb + (colbase + j * 8) / 2 + t;
        if (kf >= nf) continue;
        dst.ptr[(long long)kf * dst.ld_k + dbase + l] = make_double2(acc[i][j][2 * h] * s, acc[i][j][2 * h + 1] * s);
      }
    }
  if (zero_fill && !dst.packed && t0 == m) {
    const int nz_lo = m, nz_hi = P.lmax - lcap;  // rows [0, m) and (lcap, lmax]
    const int nrow = nz_lo + max(nz_hi, 0);
    for (int idx = tid; idx < nrow * NF; idx += 32 * kConsumerWarps) {
      const int r = idx % nrow, fl = idx / nrow, kf = kb + fl;
      if (kf >= nf) continue;
      const int l = (r < nz_lo) ? r : lcap + 1 + (r - nz_lo);
      dst.ptr[(long long)kf * dst.ld_k + (long long)m * dst.ld_m + l] = make_double2(0.0, 0.0);
    }
  }
}

template <int NCOL>
static int launch_ana_ncol(const shtb_plan* p, const void* W, int nf, int row_end, int mlim, const CoefSink& dst,
                           const Factors& F, int zero_fill, cudaStream_t st) {
  if ((p->npair + kAnaPairs - 1) / kAnaPairs > kAnaMaxChunks)
    return set_error(SHTB_ERR_UNSUPPORTED, "nlat too large for the FP64 analysis kernel");
  auto kern = leg_ana64_kernel<NCOL>;
  const size_t smem = AnaSmem<NCOL>::bytes();
  SHTB_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                "analysis smem attr");
  constexpr int NF = WarpTile<NCOL>::NF;
  dim3 grid(p->dev.natiles, (nf + NF - 1) / NF);
  prof_begin(st);
  kern<<<grid, kLegThreads, smem, st>>>(p->dev, (const double2*)W, nf, row_end, mlim, dst, F, zero_fill, p->d_err);
  SHTB_LAUNCHED("legendre analysis kernel");
  return SHTB_OK;
}

int launch_leg_ana64(const shtb_plan* p, const void* W, int nf, int row_end, int mlim, const CoefSink& dst,
                     const Factors& F, int zero_fill, cudaStream_t st) {
  if (nf <= 2) return launch_simt_ana64(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (nf > 32) return launch_ana_ncol<128>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (nf > 16) return launch_ana_ncol<64>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (nf > 8) return launch_ana_ncol<32>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  if (nf > 4) return launch_ana_ncol<16>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
  return launch_ana_ncol<8>(p, W, nf, row_end, mlim, dst, F, zero_fill, st);
}

}  // namespace shtb
