// simt.cu — Legendre stage for one or two fields, with the recurrence regenerated on the fly
// on the FP64 pipes: synthesis and analysis of the FP64 and of the mixed path.
//
// With one or two fields an MMA tile is mostly padding: the FP64 MMAs take 8 columns for 2 or
// 4, and the tensor-core GEMM of mixed.cu streams 4 bytes of P table per value for 2 or 4
// columns. Here a value of P costs 2 FP64 operations of the c-scaled three-term recurrence
//   r_l = alpha_l x r_{l-1} - r_{l-2},   P_l^m = c_l r_l
// and each field 2 more (real and imaginary part), and P is never read from memory. Chains
// start from the plan's start records (zeros below the start degree, a multiple of kStartStep
// degrees from m, so starts are looked for once every kStartStep degrees).
//   synthesis  lane = latitude pair; the sum over degrees stays in the lane
//   analysis   lane = latitude pair, 16 lanes = a segment of degrees with their sums in registers,
//              two segments a warp; the sum over pairs crosses the lanes once, at the end
// E and O (even and odd l - m) sums in FP64 on both paths. Measured at lmax 1023, one field
// (B200): FP64 synthesis 1236 -> 94 us, analysis 566 -> 135 us against the 8-column MMA
// kernels; the FP64 pipes alone would take about 60 us each. Mixed path, against the analysis GEMM,
// which streams 4 bytes a value of P (134 MB at lmax 511) for 2 or 4 columns and sums in FP32: lmax 511
// one field 41 -> 31 us, two fields 37 -> 46; lmax 1023 160 -> 135 and 164 -> 222. Two fields keep
// this kernel all the same: no P table, and FP64 sums (1.5e-7 from 64 bits at lmax 511, the GEMM 2.3e-7).
#include <climits>
#include <cstring>
#include <type_traits>

#include "kernels.cuh"

namespace shtb {
namespace sx {

constexpr int kThreads = 128;

struct Args {
  PlanDev P;
  Factors F;              // per-(l, m) multipliers of the coefficients
  const void* cin;        // synthesis: coefficients (double2 or float2); analysis: Fourier buffer
  void* out;              // synthesis: Fourier buffer; analysis: coefficients
  long long ld_k, ld_m;   // coefficient strides (field, order) and layout, as CoefSrc / CoefSink
  int packed;
  int nf, lend;           // last degree of the sums
  int mlim, lcap, zero_fill;   // analysis: largest order, last stored degree, clear l < m and l > lcap
};

template <typename C> struct Real;
template <> struct Real<double2> { using type = double; };
template <> struct Real<float2> { using type = float; };

__device__ __forceinline__ double2 wide(double2 v) { return v; }
__device__ __forceinline__ double2 wide(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ void narrow(double2& d, double2 v) { d = v; }
__device__ __forceinline__ void narrow(float2& d, double2 v) { d = make_float2((float)v.x, (float)v.y); }

__device__ __forceinline__ double factor_at(const Args& a, long long poff, int l, int m) {
  const Factors& F = a.F;
  double s = (m == 0) ? F.mf0 : F.mf1;
  if (F.fac) s *= F.fac[poff + (l - m)];
  if (F.sc_mode) {
    const double q = F.sc[l + (long long)(a.P.lmax + 1) * m];
    s = (F.sc_mode == 1) ? s * q : s / q;
  }
  return s;
}

// Offset of degree 0 of order m in one field's coefficients.
__device__ __forceinline__ long long coef_base(const Args& a, long long poff, int m) {
  return a.packed == 1 ? poff - m : a.packed == 2 ? lm_base(a.P.lmax, a.P.mres, m) : (long long)m * a.ld_m;
}

// ------------------------------------------------------------------------- synthesis
// One warp per CTA: a lane carries UP latitude pairs of one order. Per degree and field one
// broadcast 16-byte shared-memory load feeds 2 UP multiply-adds: a broadcast load still fills
// 32 lanes' registers (24 bytes a degree with alpha: 6 cycles of the SM's 128-byte path at one
// field) while a pair's 4 FP64 operations take 2 cycles of its 64 units, so one pair per lane
// is bound by those loads and four per lane by the FP64 units. The order's alpha and
// coefficients (times the factors, in FP64) are staged kChunk degrees at a time in two
// buffers; the next chunk's values are in registers while the current one is summed. Warps
// share nothing: the warps nearer the poles start at higher degrees, and in CTAs of four
// warps the barrier of the shared staging made them wait for the others (148 us, 44 % of
// the issue slots, at lmax 1023 and one field).
// 64 degrees at any field count: with 32 for two fields the next chunk's loads outlast the sums of
// the current one (synthesis of two fields from cold caches, lmax 255 20.5 -> 16.4 us, 511 38.9 -> 32.8).
constexpr int kChunk = 64;   // two degrees per lane

template <int NF, int UP>
struct SynWarp {   // one warp's shared memory
  double2 c[2][kChunk * NF];       // coefficients of two chunks
  double2 s[UP][32];               // start states
  double al[2][kChunk];
};

// Pairs 32 UP pb .. of order im.
template <typename C, int NF, int UP>
__device__ __forceinline__ void syn_item(const Args& a, int im, int pb, SynWarp<NF, UP>& sw) {
  constexpr int CH = kChunk;
  auto& sAl = sw.al;
  auto& sC = sw.c;
  auto& sS = sw.s;
  const PlanDev& P = a.P;
  const int m = im * P.mres;
  const int lane = threadIdx.x & 31;
  const int npair = P.npair, ndeg = a.lend - m + 1;
  const long long poff = P.off[im];
  const C* cin = (const C*)a.cin + coef_base(a, poff, m) + m;
  const int pair0 = pb * (32 * UP) + lane;
  double x[UP], ra[UP], rb[UP];
  int l0[UP];
  int mn = INT_MAX / 2;   // first start of the warp's pairs, relative to m (a multiple of kStartStep)
#pragma unroll
  for (int u = 0; u < UP; ++u) {
    const int pair = pair0 + 32 * u;
    const bool ok = pair < npair;
    x[u] = ok ? P.x[pair] : 0.0;
    l0[u] = ok ? P.l0[(size_t)im * npair + pair] - m : INT_MAX / 2;
    sS[u][lane] = ok ? P.start[(size_t)im * npair + pair] : make_double2(0.0, 0.0);
    ra[u] = rb[u] = 0.0;
    mn = min(mn, l0[u]);
  }
  mn = __reduce_min_sync(0xffffffffu, mn);
  double2 accE[UP][NF], accO[UP][NF];
#pragma unroll
  for (int u = 0; u < UP; ++u)
#pragma unroll
    for (int k = 0; k < NF; ++k) accE[u][k] = accO[u][k] = make_double2(0.0, 0.0);

  // chunk stager: lane stages degrees lane and lane + 32 of every field
  double al[2], cf[2];
  C cv[2][NF];
  auto fetch = [&](int d0) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int d = d0 + lane + 32 * q;
      al[q] = cf[q] = 0.0;
#pragma unroll
      for (int k = 0; k < NF; ++k) cv[q][k].x = cv[q][k].y = 0;
      if (d < ndeg) {
        al[q] = P.alpha[poff + d];
#pragma unroll
        for (int k = 0; k < NF; ++k) cv[q][k] = cin[(long long)k * a.ld_k + d];
        cf[q] = factor_at(a, poff, m + d, m);
      }
    }
  };
  auto put = [&](int b) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int sd = lane + 32 * q;
      sAl[b][sd] = al[q];
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        const double2 c = wide(cv[q][k]);
        sC[b][sd * NF + k] = make_double2(c.x * cf[q], c.y * cf[q]);
      }
    }
  };
  int buf = 0;
  if (mn < ndeg) {
    fetch(mn);
    put(0);
  }
  __syncwarp();
  for (int d0 = mn; d0 < ndeg; d0 += CH, buf ^= 1) {
    const bool more = d0 + CH < ndeg;
    if (more) fetch(d0 + CH);
    const int nd = min(CH, ndeg - d0);
    auto step = [&](int d, double2 (&acc)[UP][NF]) {
      const double av = sAl[buf][d];
      double2 c[NF];
#pragma unroll
      for (int k = 0; k < NF; ++k) c[k] = sC[buf][d * NF + k];
#pragma unroll
      for (int u = 0; u < UP; ++u) {
        const double r = fma(av * x[u], ra[u], -rb[u]);
        rb[u] = ra[u];
        ra[u] = r;
#pragma unroll
        for (int k = 0; k < NF; ++k) {
          acc[u][k].x = fma(r, c[k].x, acc[u][k].x);
          acc[u][k].y = fma(r, c[k].y, acc[u][k].y);
        }
      }
    };
    for (int g = 0; g < nd; g += kStartStep) {
      bool st = false;
#pragma unroll
      for (int u = 0; u < UP; ++u) st |= l0[u] == d0 + g;
      if (__any_sync(0xffffffffu, st)) {
#pragma unroll
        for (int u = 0; u < UP; ++u)
          if (l0[u] == d0 + g) {
            const double2 v = sS[u][lane];
            ra[u] = v.x;
            rb[u] = v.y;
          }
      }
      // degrees past the order's last have zero alpha and coefficients
#pragma unroll
      for (int d = 0; d < kStartStep; d += 2) {
        step(g + d, accE);
        step(g + d + 1, accO);
      }
    }
    if (more) {
      put(buf ^ 1);
      __syncwarp();
    }
  }
#pragma unroll
  for (int u = 0; u < UP; ++u) {
    const int pair = pair0 + 32 * u;
    if (pair >= npair) continue;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
      C* w = (C*)a.out + (((size_t)k * P.nm + im) * 2) * npair + pair;
      narrow(w[0], accE[u][k]);
      narrow(w[npair], accO[u][k]);
    }
  }
}

template <typename C, int NF, int UP>
__global__ void __launch_bounds__(32) syn_kernel(const __grid_constant__ Args a) {
  __shared__ __align__(16) SynWarp<NF, UP> sw;
  syn_item<C, NF, UP>(a, blockIdx.y, blockIdx.x, sw);
}

// -------------------------------------------------------------------------- analysis
// a_l = sum over pairs of P_l(x_pair) W[pair]: kLanes lanes own a segment of kSeg<NF> = 32 / NF
// consecutive degrees of one order and hold their sums in every lane (kSeg x NF complex doubles
// = 128 registers); lane = latitude pair, a warp's kSplit consecutive segments (a span) walk the
// pairs together, kLanes at a time, and share the lines they read. Per pair and segment the chain
// starts from the plan's checkpoint and the pair's Fourier values stay in registers, so P
// costs 2 FP64 operations and each field 2 more, with one broadcast load of alpha per degree.
// The lanes' sums meet once, at the end, in a butterfly that halves the values each lane keeps
// per step and leaves lane j of a segment with items kSplit j .. (item i = degree i / NF, field
// i % NF): 30 exchanges for two segments, 31 for one where a segment has all 32 lanes (32 uneven
// transforms 602 -> 575 us, lmax 1023 and one field 156 -> 152 us).
// Pair blocks whose every pair starts above the span are skipped while they lead.
// Every lane copies its own operands of the next pairs into its slots of a shared-memory
// ring (cp.async; only the lane itself reads them, so no barrier): the registers left beside
// the sums allow two warps per scheduler, too few to cover the loads. A slot holds kPU
// blocks of kLanes pairs, summed together: one alpha load serves both, and their chains overlap
// (two fields at lmax 1023 297 -> 247 us against one block). The addresses were most of the other
// instructions (12 integer ones a copy): blocks that lie inside the rows are copied from pointers that
// advance with them, and only the last block of a row, or a span that ends early, checks each
// lane's pair (247 -> 222 us; one field 150 -> 135).
template <int NF>
constexpr int kSeg = 32 / NF;
constexpr int kLanes = 16, kSplit = 32 / kLanes;
template <int NF>
constexpr int kSpan = kSplit * kSeg<NF>;
template <int NF>
constexpr int kAlLd = kSeg<NF> + 1;   // stride of a segment's alpha in shared memory: segments of a warp in other banks
constexpr int kPU = 2;
constexpr int kRing = 3;

// A warp of the persistent kernel takes up to kMaxSpans consecutive spans: the ring runs on
// into the next span's first pairs while the sums of the current one cross the lanes (32
// uneven transforms 652 -> 631 us). A single transform's warps take one: four made the CTAs
// uneven (lmax 1023, one field 154 -> 183 us, with 32 lanes a segment).
constexpr int kMaxSpans = 2;

template <typename C, int NF>
struct Ring {   // one warp's slots
  struct Slot {
    double2 ck[kPU][32];
    C w[kPU][2 * NF][32];
    double x[kPU][32];
    int l0[kPU][32];
  } s[kRing];
  int p0[kMaxSpans];   // first pair of each span of the warp
};

// Alpha and factors of a warp's spans: they load while its first operands do.
template <int NF, int MAXS>
struct SegTables {
  double al[MAXS * kSplit * kAlLd<NF>];
  double fac[MAXS * kSpan<NF>];
};

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
// Zeros unless ok; src is readable either way.
template <int BYTES>
__device__ __forceinline__ void cp_async_if(void* dst, const void* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst), n = ok ? BYTES : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(BYTES), "r"(n) : "memory");
}

template <typename C, int NF, int MAXS>
__device__ __forceinline__ void ana_segments(const Args& a, int im, int lseg0, int nsegs, SegTables<NF, MAXS>& T,
                                             Ring<C, NF>& R) {
  const int nseg = MAXS == 1 ? 1 : nsegs;
  constexpr int SG = kSeg<NF>, SP = kSpan<NF>, PU = kPU, RG = kRing;
  const PlanDev& P = a.P;
  const int lane = threadIdx.x & 31, h = lane / kLanes, j = lane % kLanes, npair = P.npair, m = im * P.mres;
  const long long poff = P.off[im];
  const int cs = P.ckstep;
  const double2* ck0 = P.ckpt + (size_t)P.ckbase[im] * npair;
  const int* pl0 = P.l0 + (size_t)im * npair;
  const C* W = (const C*)a.cin + (size_t)im * 2 * npair;
  const size_t wld = (size_t)P.nm * 2 * npair;
  const double* px = P.x;
  const int nf = a.nf;
  // each span's pairs start at the first block with a start below the span's end
  const int first = npair <= 32 ? 0 : first_live_pair(pl0, npair, lseg0 + SP);
  if constexpr (MAXS > 1) {
    for (int i = 1; i < nseg; ++i) {
      const int p = first_live_pair(pl0, npair, lseg0 + SP * (i + 1));
      if (lane == 0) R.p0[i] = p;
    }
    __syncwarp();
  }
  // next span, first pair of the next blocks and slot to copy; this lane's pointers into every row
  int fs = 0, fb = first, fq = 0;
  bool live = false, full = false;   // this lane's segment, every lane's segment holds degrees
  const double2* gck;
  const double* gx;
  const int* gl;
  const C* gw[2 * NF];
  auto seek = [&](int span, int pair) {
    const int lf = lseg0 + SP * span + SG * h;
    live = lf <= a.lend;   // the last span may hold fewer segments
    full = lseg0 + SP * span + SG * (kSplit - 1) <= a.lend;
    fb = pair;
    gck = (live ? ck0 + (size_t)((lf - m) / cs) * npair : ck0) + pair + j;
    gx = px + pair + j;
    gl = pl0 + pair + j;
#pragma unroll
    for (int r = 0; r < 2 * NF; ++r) gw[r] = W + (r >> 1) * wld + (r & 1) * npair + pair + j;
  };
  seek(0, first);
  auto fetch = [&]() {
    if constexpr (MAXS > 1) {
      while (fs < nseg && fb >= npair) {
        ++fs;
        if (fs < nseg) seek(fs, R.p0[fs]);
      }
    }
    if (MAXS == 1 || fs < nseg) {
      auto& S = R.s[fq];
      if (full && fb + kLanes * PU <= npair) {
#pragma unroll
        for (int u = 0; u < PU; ++u) {
          cp_async<16>(&S.ck[u][lane], gck + kLanes * u);
          cp_async<8>(&S.x[u][lane], gx + kLanes * u);
          cp_async<4>(&S.l0[u][lane], gl + kLanes * u);
#pragma unroll
          for (int r = 0; r < 2 * NF; ++r) cp_async<sizeof(C)>(&S.w[u][r][lane], gw[r] + kLanes * u);
        }
      } else if (fb < npair) {
#pragma unroll
        for (int u = 0; u < PU; ++u) {
          const bool ok = live && fb + j + kLanes * u < npair;
          const int d = ok ? kLanes * u : -(fb + j);   // else each row's first entry
          cp_async_if<16>(&S.ck[u][lane], gck + d, ok);
          cp_async_if<8>(&S.x[u][lane], gx + d, ok);
          cp_async_if<4>(&S.l0[u][lane], gl + d, ok);
#pragma unroll
          for (int r = 0; r < 2 * NF; ++r) cp_async_if<sizeof(C)>(&S.w[u][r][lane], gw[r] + d, ok);
        }
      }
      fb += kLanes * PU;
      gck += kLanes * PU;
      gx += kLanes * PU;
      gl += kLanes * PU;
#pragma unroll
      for (int r = 0; r < 2 * NF; ++r) gw[r] += kLanes * PU;
      fq = fq + 1 == RG ? 0 : fq + 1;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < RG - 1; ++i) fetch();
  for (int i = lane; i < nseg * SP; i += 32) {
    const int l = lseg0 + i;
    T.al[i / SG * kAlLd<NF> + i % SG] = l <= a.lend ? P.alpha[poff + (l - m)] : 0.0;
    if (l <= a.lcap) T.fac[i] = factor_at(a, poff, l, m);
  }
  __syncwarp();
  int q = 0;
  for (int seg = 0; seg < nseg; ++seg) {
    const int lseg = lseg0 + SP * seg + SG * h, roll = lseg <= a.lend ? (lseg - m) % cs : 0;
    const double* sal = T.al + kAlLd<NF> * (kSplit * seg + h);
    double2 acc[SG][NF];
#pragma unroll
    for (int s = 0; s < SG; ++s)
#pragma unroll
      for (int k = 0; k < NF; ++k) acc[s][k] = make_double2(0.0, 0.0);
    for (int p0 = seg == 0 ? first : R.p0[seg]; p0 < npair; p0 += kLanes * PU) {
      fetch();
      asm volatile("cp.async.wait_group %0;\n" ::"n"(RG - 1) : "memory");
      double x[PU], ra[PU], rb[PU];
      int l0[PU];
      double2 E[PU][NF], O[PU][NF];
      bool st = false;
      const auto& S = R.s[q];
#pragma unroll
      for (int u = 0; u < PU; ++u) {
        x[u] = S.x[u][lane];
        const double2 v = S.ck[u][lane];
        ra[u] = v.x;
        rb[u] = v.y;
        l0[u] = S.l0[u][lane];   // 0 for pairs past the end and dead segments: no start to look for
        st |= l0[u] > lseg && l0[u] < lseg + SG;
#pragma unroll
        for (int k = 0; k < NF; ++k) {
          E[u][k] = wide(S.w[u][2 * k][lane]);
          O[u][k] = wide(S.w[u][2 * k + 1][lane]);
        }
      }
      q = q + 1 == RG ? 0 : q + 1;
      auto step = [&](int s, double al) {
#pragma unroll
        for (int u = 0; u < PU; ++u) {
          const double r = fma(al * x[u], ra[u], -rb[u]);
          rb[u] = ra[u];
          ra[u] = r;
#pragma unroll
          for (int k = 0; k < NF; ++k) {
            const double2 w = (s & 1) ? O[u][k] : E[u][k];
            acc[s][k].x = fma(r, w.x, acc[s][k].x);
            acc[s][k].y = fma(r, w.y, acc[s][k].y);
          }
        }
      };
      if (!__any_sync(0xffffffffu, st || roll)) {
#pragma unroll
        for (int s = 0; s < SG; ++s) step(s, sal[s]);
      } else {
        // a pair of the warp starts inside the segment, or the checkpoint lies below it
        double2 v[PU];
#pragma unroll
        for (int u = 0; u < PU; ++u) {
          const int p = p0 + kLanes * u + j;
          v[u] = p < npair ? P.start[(size_t)im * npair + p] : make_double2(0.0, 0.0);
        }
        auto begin = [&](int l) {
#pragma unroll
          for (int u = 0; u < PU; ++u)
            if (l == l0[u]) {
              ra[u] = v[u].x;
              rb[u] = v[u].y;
            }
        };
        for (int l = lseg - roll; l < lseg; ++l) {
          begin(l);
          const double al = P.alpha[poff + (l - m)];
#pragma unroll
          for (int u = 0; u < PU; ++u) {
            const double r = fma(al * x[u], ra[u], -rb[u]);
            rb[u] = ra[u];
            ra[u] = r;
          }
        }
#pragma unroll
        for (int s = 0; s < SG; ++s) {
          if (s % kStartStep == 0) begin(lseg + s);
          step(s, sal[s]);
        }
      }
    }
    // items i = s * NF + k; after the step with lane bit o, a lane keeps the half of its items
    // whose index has bit o * kSplit as its lane number has bit o
    double2 (&v)[SG * NF] = reinterpret_cast<double2 (&)[SG * NF]>(acc);
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) {
      const bool up = j & o;
#pragma unroll
      for (int i = 0; i < o * kSplit; ++i) {
        const double2 send = up ? v[i] : v[i + o * kSplit], keep = up ? v[i + o * kSplit] : v[i];
        v[i].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, o);
        v[i].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, o);
      }
    }
#pragma unroll
    for (int i = 0; i < kSplit; ++i) {
      const int l = lseg + (j * kSplit + i) / NF, k = (j * kSplit + i) % NF;
      if (l <= a.lcap && k < nf) {
        const double f = T.fac[l - lseg0];
        C* dst = (C*)a.out + (long long)k * a.ld_k + coef_base(a, poff, m) + l;
        narrow(*dst, make_double2(v[i].x * f, v[i].y * f));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");   // no copy in flight past the last segment
}

// CTA = kAnaWarps consecutive spans of one order, a warp each: blockIdx.y of NF parts of a tile
// of kSimtTile degrees.
constexpr int kAnaWarps = 2;
template <typename C, int NF>
__global__ void __launch_bounds__(32 * kAnaWarps) ana_kernel(const __grid_constant__ Args a) {
  constexpr int ND = kAnaWarps * kSpan<NF>;
  __shared__ SegTables<NF, 1> tab[kAnaWarps];
  __shared__ __align__(16) Ring<C, NF> ring[kAnaWarps];
  const PlanDev& P = a.P;
  const int2 tile = P.stiles[blockIdx.x];
  const int im = tile.x, t0 = tile.y + ND * blockIdx.y, m = im * P.mres;
  if (m > a.mlim || t0 > a.lend) return;
  const int w = threadIdx.x >> 5, lseg = t0 + kSpan<NF> * w;
  if (lseg <= a.lend) ana_segments<C, NF, 1>(a, im, lseg, 1, tab[w], ring[w]);
  if (a.zero_fill && t0 == m) {
    const int nrow = m + max(P.lmax - a.lcap, 0);   // rows [0, m) and (lcap, lmax]
    for (int idx = threadIdx.x; idx < nrow * a.nf; idx += blockDim.x) {
      const int r = idx % nrow, k = idx / nrow, l = (r < m) ? r : a.lcap + 1 + (r - m);
      narrow(((C*)a.out)[(long long)k * a.ld_k + (long long)m * a.ld_m + l], make_double2(0.0, 0.0));
    }
  }
}

// Persistent synthesis over the items of many transforms (uneven batches), one item per warp:
// item = (transform, order index, block of 32 kGroupUP latitude pairs), list sorted by
// decreasing work and claimed by each warp from the device counter *queue (zero at launch). An
// item is one CTA's work of syn_kernel, so the results are the same bit for bit (two pairs per
// lane and chunks fetched ahead: 32 uneven transforms 631 -> 602 us against one pair per lane
// and a wait for each chunk).
constexpr int kGroupUP = 2;
union GroupSynWarp {
  SynWarp<1, kGroupUP> s1;
  SynWarp<2, kGroupUP> s2;
};

__global__ void __launch_bounds__(kThreads, 4) syn_group_kernel(const Args* __restrict__ targs,
                                                                const int4* __restrict__ items, int nitems,
                                                                int* __restrict__ queue,
                                                                unsigned long long* __restrict__ t0) {
  __shared__ __align__(16) GroupSynWarp sw[kThreads / 32];
  group_start(t0);
  GroupSynWarp& w = sw[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  for (;;) {
    int i = 0;
    if (lane == 0) i = atomicAdd(queue, 1);
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= nitems) break;
    const int4 it = items[i];
    const Args& a = targs[it.x];
    __syncwarp();   // the previous item's shared memory is read
    if (a.nf == 1)
      syn_item<float2, 1, kGroupUP>(a, it.y, it.z, w.s1);
    else
      syn_item<float2, 2, kGroupUP>(a, it.y, it.z, w.s2);
  }
}

// Persistent analysis over the items of many transforms, one item per warp: item = (transform,
// order, first span, spans), list sorted by decreasing work and claimed by
// each warp from *queue. A span's sums are those of ana_kernel, so the results are the same bit for bit. The
// warp of an order's first span clears the degrees below the order. done[t] receives the
// largest %globaltimer value at which an item of transform t was stored.
struct GroupAnaWarp {
  union {
    Ring<float2, 1> r1;
    Ring<float2, 2> r2;
  };
  union {
    SegTables<1, kMaxSpans> t1;
    SegTables<2, kMaxSpans> t2;
  };
};

template <int NF>
__device__ __forceinline__ void ana_warp_item(const Args& a, int im, int seg, int nseg, Ring<float2, NF>& R,
                                              SegTables<NF, kMaxSpans>& T) {
  const int lane = threadIdx.x & 31, m = im * a.P.mres, lseg = m + kSpan<NF> * seg;
  __syncwarp();   // the previous item's tables are read
  ana_segments<float2, NF, kMaxSpans>(a, im, lseg, nseg, T, R);
  if (seg == 0)
    for (int k = 0; k < a.nf; ++k) {
      float2* col = (float2*)a.out + (long long)k * a.ld_k + (long long)m * a.ld_m;
      for (int l = lane; l < m; l += 32) col[l] = make_float2(0.f, 0.f);
    }
}

__global__ void __launch_bounds__(32 * kAnaWarps) ana_group_kernel(const Args* __restrict__ targs,
                                                             const int4* __restrict__ items, int nitems,
                                                             int* __restrict__ queue,
                                                             unsigned long long* __restrict__ done) {
  __shared__ __align__(16) GroupAnaWarp sw[kAnaWarps];
  GroupAnaWarp& w = sw[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  for (;;) {
    int i = 0;
    if (lane == 0) i = atomicAdd(queue, 1);
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= nitems) break;
    const int4 it = items[i];
    const Args& a = targs[it.x];
    if (a.nf == 1)
      ana_warp_item<1>(a, it.y, it.z, it.w, w.r1, w.t1);
    else
      ana_warp_item<2>(a, it.y, it.z, it.w, w.r2, w.t2);
    __syncwarp();
    if (lane == 0) atomicMax(done + it.x, group_time());
  }
}

}  // namespace sx

// ---------------------------------------------------------------------------- host
bool simt_applicable(const shtb_plan*, int nf) { return nf >= 1 && nf <= 2; }

static sx::Args simt_args(const shtb_plan* p, const void* in, void* out, const Factors& F, int nf, int lend) {
  sx::Args a{};
  a.P = p->dev;
  a.F = F;
  a.cin = in;
  a.out = out;
  a.nf = nf;
  a.lend = lend;
  return a;
}

// Pairs per lane: two (94 us at lmax 1023, one field; four 96 us) where that still gives every
// SM a dozen warps, else one.
static int syn_pairs_per_thread(const shtb_plan* p, int nmu) {
  const long long per32 = (long long)((p->npair + 31) / 32) * nmu;
  return per32 / 2 >= 12ll * p->nsm ? 2 : 1;
}

template <typename C, int NF>
static int launch_syn(const shtb_plan* p, const sx::Args& a, int nmu, const char* name, cudaStream_t st) {
  const int up = syn_pairs_per_thread(p, nmu);
  const dim3 grid((p->npair + 32 * up - 1) / (32 * up), nmu);
  prof_begin(st);
  if (up == 2)
    sx::syn_kernel<C, NF, 2><<<grid, 32, 0, st>>>(a);
  else
    sx::syn_kernel<C, NF, 1><<<grid, 32, 0, st>>>(a);
  SHTB_LAUNCHED(name);
  return SHTB_OK;
}

template <typename C, int NF>
static int launch_ana(const shtb_plan* p, const sx::Args& a, const char* name, cudaStream_t st) {
  static_assert(sx::kAnaWarps * sx::kSpan<NF> * NF == kSimtTile, "tile list of the plan");
  prof_begin(st);
  sx::ana_kernel<C, NF><<<dim3(p->dev.nstiles, NF), 32 * sx::kAnaWarps, 0, st>>>(a);
  SHTB_LAUNCHED(name);
  return SHTB_OK;
}

static Factors mixed_factors(const shtb_plan* p, int sc_mode) {
  return Factors{p->dev.cfac, p->d_scale, p->d_scale ? sc_mode : 0, 1.0, 1.0};
}

// Coefficients (FP32, dense or packed LM) -> Fourier buffer W (FP32), orders 0..mlim.
int launch_simt_syn(const shtb_plan* p, const void* alm, void* W, int nf, int ltr, int mlim, int packed,
                    cudaStream_t st) {
  sx::Args a = simt_args(p, alm, W, mixed_factors(p, 1), nf, ltr);
  a.packed = packed ? 2 : 0;
  a.ld_k = packed ? lm_count(p->lmax, p->mmax, p->mres) : (long long)(p->lmax + 1) * (p->mmax + 1);
  a.ld_m = p->lmax + 1;
  const int nmu = mlim / p->mres + 1;
  return nf == 1 ? launch_syn<float2, 1>(p, a, nmu, "simt legendre synthesis kernel", st)
                 : launch_syn<float2, 2>(p, a, nmu, "simt legendre synthesis kernel", st);
}

// Fourier buffer W (FP32) -> coefficients (FP32, dense or packed LM), degrees up to ltr.
int launch_simt_ana(const shtb_plan* p, const void* W, void* alm, int nf, int ltr, int mlim, int packed,
                    cudaStream_t st) {
  sx::Args a = simt_args(p, W, alm, mixed_factors(p, 2), nf, ltr);
  a.packed = packed ? 2 : 0;
  a.ld_k = packed ? lm_count(p->lmax, p->mmax, p->mres) : (long long)(p->lmax + 1) * (p->mmax + 1);
  a.ld_m = p->lmax + 1;
  a.mlim = mlim;
  a.lcap = ltr;
  a.zero_fill = !packed;
  return nf == 1 ? launch_ana<float2, 1>(p, a, "simt legendre analysis kernel", st)
                 : launch_ana<float2, 2>(p, a, "simt legendre analysis kernel", st);
}

// FP64 coefficients -> Fourier buffer for one or two fields.
int launch_simt_syn64(const shtb_plan* p, const CoefSrc& src, const Factors& F, void* W, int nf, int row_end, int mlim,
                      cudaStream_t st) {
  sx::Args a = simt_args(p, src.ptr, W, F, nf, std::min(row_end, p->lrec));
  a.packed = src.packed;
  a.ld_k = src.ld_k;
  a.ld_m = src.ld_m;
  const int nmu = mlim / p->mres + 1;
  return nf == 1 ? launch_syn<double2, 1>(p, a, nmu, "legendre synthesis kernel", st)
                 : launch_syn<double2, 2>(p, a, nmu, "legendre synthesis kernel", st);
}

// FP64 Fourier buffer -> coefficients for one or two fields.
int launch_simt_ana64(const shtb_plan* p, const void* W, int nf, int row_end, int mlim, const CoefSink& dst,
                      const Factors& F, int zero_fill, cudaStream_t st) {
  sx::Args a = simt_args(p, W, dst.ptr, F, nf, std::min(row_end, p->lrec));
  a.packed = dst.packed;
  a.ld_k = dst.ld_k;
  a.ld_m = dst.ld_m;
  a.mlim = mlim;
  a.lcap = dst.packed == 1 ? a.lend : std::min(a.lend, p->lmax);
  a.zero_fill = zero_fill && !dst.packed;
  return nf == 1 ? launch_ana<double2, 1>(p, a, "legendre analysis kernel", st)
                 : launch_ana<double2, 2>(p, a, "legendre analysis kernel", st);
}

// ------------------------------------------------------------- grouped transforms
size_t simt_args_bytes() { return sizeof(sx::Args); }

void simt_fill_args(const shtb_plan* p, int syn, const void* in, void* out, int nf, void* host_args) {
  sx::Args a = simt_args(p, in, out, mixed_factors(p, syn ? 1 : 2), nf, p->lmax);
  a.ld_k = (long long)(p->lmax + 1) * (p->mmax + 1);
  a.ld_m = p->lmax + 1;
  a.lcap = p->lmax;
  std::memcpy(host_args, &a, sizeof(a));
}

int simt_ana_span(int nf) { return nf == 1 ? sx::kSpan<1> : sx::kSpan<2>; }

// Several once every warp slot (two per scheduler) has work for three rounds.
int simt_ana_spans_per_warp(long long spans, int nsm) {
  return (int)std::max(1ll, std::min<long long>(sx::kMaxSpans, spans / (3ll * nsm * 8)));
}

int simt_syn_pair_blocks(const shtb_plan* p) {   // per-warp items of the group kernel
  return (p->npair + 32 * sx::kGroupUP - 1) / (32 * sx::kGroupUP);
}

int launch_simt_group(const void* targs, const int4* items, int nitems, int grid, int* queue, unsigned long long* t0,
                      cudaStream_t st) {
  if (nitems <= 0) return SHTB_OK;
  sx::syn_group_kernel<<<grid, sx::kThreads, 0, st>>>((const sx::Args*)targs, items, nitems, queue, t0);
  count_launch();
  SHTB_TRY_CUDA(cudaGetLastError(), "simt group launch");
  return SHTB_OK;
}

int launch_simt_ana_group(const void* targs, const int4* items, int nitems, int grid, int* queue,
                          unsigned long long* done, cudaStream_t st) {
  if (nitems <= 0) return SHTB_OK;
  sx::ana_group_kernel<<<grid, 32 * sx::kAnaWarps, 0, st>>>((const sx::Args*)targs, items, nitems, queue, done);
  count_launch();
  SHTB_TRY_CUDA(cudaGetLastError(), "simt analysis group launch");
  return SHTB_OK;
}

}  // namespace shtb
