// Direct TSQR + Householder reconstruction of a panel at most kDirectB (32)
// columns wide, FP64, with a fan-in-4 reduction tree and compact-WY Q blocks.
//
// Reference path: alg/QR/hh_recon/hh_recon.cxx:129-321 with the TSQR of
// alg/QR/tsqr/bitree_tsqr.cxx:91-248 and the Q1 construction of
// alg/QR/tsqr/construct_tsqr_Q.cxx:34-242.  The reference pairs ranks in a
// binary tree and forms Q1 by applying every node's reflectors (dtprfb) and
// every leaf's reflectors (dormqr) to [I; 0].  On GB300 the FP64 pipe is
// narrow (about 2 DFMA/clk/SM) and every Householder step is a chain of
// dependent FP64 operations and block barriers, so the design minimises the
// number of sequential steps on the critical path:
//  * leaves of at most leaf_rows rows, one CTA each: b Householder steps in
//    the critical-warp schedule below, then the leaf's compact-WY T (T^-1
//    from the Gram matrix V^T V);
//  * a fan-in-4 tree: the node stacks up to four R factors and runs b
//    Householder steps on the stacked matrix (the zeros below the children's
//    diagonals stay zero); with V = [I; V_2..V_4] the node's Q blocks are
//    Q_1 = I - T and Q_k = -V_k T (all upper triangular), so no explicit-Q
//    pass is needed.  Two schedules: k_hr6_pipe, where every node is a CTA
//    that starts column j as soon as its children have published it (the
//    levels overlap; roles by atomic ticket, bounded waits), and
//    k_hr4_leaf_tree, where the last CTA to arrive combines a node;
//  * the root: Q1_top = (I - V0 T0 V0^T) Q_1^(1) ... Q_1^(depth) on the top
//    b rows, then the sign-choice LU of Q1_top - S, and L\(S R), T, W and
//    U^-1.  In k_hr6_pipe leaf 0 and the nodes on its path build Q1_top as a
//    prefix product while they finish, and one extra CTA solves the root;
//  * Y = (I - V T V_top^T) (Q^(1) ... Q^(depth)) U^-1 per leaf, the Q blocks
//    taken along the leaf's path: beside the tree where its CTAs find free
//    SMs (k_hr6_y), in a launch of its own otherwise (k_hr4_form_y).
// The Householder factor is canonical, so the result equals the binary-tree
// reconstruction and LAPACK's dgeqrf up to rounding.
#include <math.h>

#include <algorithm>

#include "kernels.cuh"

namespace candmc {

constexpr int kFan = 4;

// Target rows per TSQR leaf (tuning knob, candmc_set_tuning("leaf_rows", v));
// 0: chosen by the panel's height (hr_direct4).
int64_t g_leaf_rows = 0;
// Leaf height of latency-bound panels.  A leaf's step is bound by the FP64
// pipe from 128 rows on; below, by its chain.  8192 x 32 takes 194 us with
// 128-row leaves, 240 with 64 rows (its CTAs share SMs) and 252 with 256.
constexpr int64_t kLeafRows = 128;
int64_t g_pipe_leaf_rows = 0;   // the lookahead's panels (knob "pipe_leaf_rows"); 0: as without it
thread_local int64_t t_leaf_rows = 0;
// Pipelined tree on/off (tuning knob, candmc_set_tuning("pipe_tree", 0|1)).
int g_pipe_tree = 1;

__device__ __forceinline__ int64_t t4_leaf_row0(int64_t m, int P, int i) {
  return (m / P) * i + (m % P) * i / P;
}

// ---- Householder QR of a shared-memory block, critical-warp schedule.
//
// What bounds it: a warp-wide FP64 instruction (fma, add, mul, compare or
// conversion alike, whatever lanes are active) takes 65 cycles of its SM
// sub-partition's FP64 pipe and 65 cycles of latency (measured), so the unit
// of cost is the FP64 instruction: per sub-partition for throughput, per
// dependent chain for latency.  The schedule therefore
//  * gives one warp (warp 0, alone with the memory warps on its sub-partition)
//    the serial chain: apply reflector j-1 to column j, form reflector j;
//  * spreads the other columns over six warps on the other three
//    sub-partitions, two warps each, so that one's shuffles and loads hide
//    behind the other's arithmetic;
//  * keeps the reflectors unnormalised: H = I - gamma v v^T with
//    v = (alpha - beta, x), gamma = 1 / (q + |alpha| sigma), q = alpha^2 + |x|^2,
//    sigma = sqrt(q), beta = -sign(alpha) sigma (LAPACK dlarfg's beta), which
//    takes the division by alpha - beta and the scaling of x off the chain;
//    the tails are divided by their heads once, after the last column;
//  * seeds sigma and gamma with FP32 approximations exchanged by integer
//    operations (a conversion would cost an FP64 slot) and refines them by one
//    third-order step;
//  * forms T from the Gram matrix of the finished reflectors, after the last
//    column of R has been published.
// One column step of a 64-row leaf takes about 30 FP64 instructions of chain
// (2.1 k cycles) instead of two normalised passes with FP64-pipe conversions.
// An all-zero tail takes v = e_j, gamma = 2, beta = -alpha (a sign flip), the
// convention of the reconstruction, so that T^-1 = striu(V^T V) +
// diag(V^T V) / 2 (alg/QR/qr_2d/qr_2d.cxx:22-60) holds for every reflector.
// This thread's warp, in a form the compiler knows to be uniform: branches on
// it (and on columns derived from it) become plain jumps instead of divergent
// regions, worth 20 % of a column step.
__device__ __forceinline__ int warp_id() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

constexpr int kLeafThreads = 288;   // 9 warps: the critical one, 6 for the columns, 2 for memory
constexpr int kPollWarp = 4;        // sub-partition 0: waits for the children's columns; a column warp in leaves
constexpr int kPubWarp = 8;         // sub-partition 0: publishes finished columns
constexpr int kBulkWarps = 6;       // warps 1-3 and 5-7
constexpr int kLd = kDirectB + 1;   // leading dimension of the 32 x 32 shared blocks
constexpr int kMaxR = 8;            // rows per lane: leaves of up to 256 rows, nodes of 4 x 32
// leaves from which the Y formation takes its path products from a top-down
// pass over the nodes instead of multiplying each leaf's whole path itself
constexpr int kNodeMinLeaves = 256;
// rows from which panels take 256-row leaves (65536 x 32: 680 us against 766
// with 128-row leaves; 262144 x 32: 1866 against 2361)
constexpr int64_t kTallPanelRows = 32768;

// Index 0..5 of a column warp (1-3, 5-7), 6 for the seventh warp of a leaf (4,
// beside the critical one), or -1.
__device__ __forceinline__ int bulk_index(int warp) {
  return (warp >= 1 && warp <= 3) ? warp - 1 : (warp >= 5 && warp <= 7) ? warp - 2 : warp == kPollWarp ? 6 : -1;
}

// The columns of a block over its warps.  While many columns are left, the six
// column warps bound a step and the critical warp's sub-partition has time to
// spare, so warp 6 takes the columns 4, 9, 14 and 19, which are finished before
// the chain bounds the steps; the other 28, in order, go round the six
// (slot i = q + 6 k of warp q).
__device__ __forceinline__ int leaf_col(int q, int k) {
  const int i = q + kBulkWarps * k, g = i >> 2;
  return q == kBulkWarps ? (k < 4 ? 5 * k + 4 : kDirectB) : i + (g < 4 ? g : 4);
}
// the first k with leaf_col(q, k) >= c
__device__ __forceinline__ int leaf_first(int q, int c) {
  if (q == kBulkWarps) return c / 5 < 4 ? c / 5 : 4;
  const int g = c / 5, i = c - (g < 4 ? g : 4) - q;   // slots of the columns before c
  return i > 0 ? (i + kBulkWarps - 1) / kBulkWarps : 0;
}

// Sums over the warp of N values per lane (N a power of two): lanes
// k (32 / N) .. (k + 1) (32 / N) - 1 return sum number k.  Halving the values
// and the lanes together takes N - 1 + 5 - log2(N) additions instead of 5 N.
template <int N>
__device__ __forceinline__ double warp_sum_held(double (&d)[N]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < n / 2; ++k)
      d[k] = (up ? d[k + n / 2] : d[k]) + __shfl_xor_sync(0xffffffffu, up ? d[k] : d[k + n / 2], o);
    o >>= 1;
  }
  double s = d[0];
#pragma unroll
  for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// barrier `id` of n threads (a multiple of 32)
__device__ __forceinline__ void named_bar(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Polls before a bounded wait gives up (tuning knobs "panel_polls": on another CTA
// of the panel; "panel_smem_polls": on another warp of the CTA).  About 100 ns each.
int g_panel_polls = 1 << 22;
int g_panel_smem_polls = 1 << 22;
constexpr int kStepThreads = 7 * 32;   // the critical warp and the six column warps of a node
constexpr int kLeafStepThreads = 8 * 32;   // those of a leaf, with the seventh
constexpr int kStepBar = 3;            // their barrier, one per column step
constexpr int kGamBar = 4;             // the critical warp arrives when gamma is written, the others wait
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__device__ __forceinline__ int hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }
// x with its sign flipped when `neg` is set
__device__ __forceinline__ double flip_if(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? 0x80000000 : 0), __double2loint(x));
}
// FP32 value of a positive double with exponent within +-100 (truncated), and back
__device__ __forceinline__ float f32_of(double x) {
  return __int_as_float(__funnelshift_l(__double2loint(x), __double2hiint(x) - 0x38000000, 3));
}
__device__ __forceinline__ double f64_of(float x) {
  const int i = __float_as_int(x);
  return __hiloint2double((i >> 3) + 0x38000000, i << 29);
}

// 1 / x: an FP32 seed (relative error below 2^-20) and one third-order step,
// e = 1 - x y, y (1 + e + e^2), whose error e^3 lies below 2^-60.
__device__ __forceinline__ double quick_rcp(double x) {
  const int h = hi_abs(x);
  if (h < ((1023 - 90) << 20) || h >= ((1023 + 90) << 20)) return 1.0 / x;
  const double y = flip_if(f64_of(__fdividef(1.0f, f32_of(fabs(x)))), __double2hiint(x) < 0);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// The scalars of one reflector from alpha and q = alpha^2 + |x|^2: sigma =
// sqrt(q) as q r (1 + e/2 + 3 e^2/8) with e = 1 - q r^2 (the series' next
// term is below 2^-62), h = alpha + sign(alpha) sigma, gamma = 1 / (q + |alpha|
// sigma).  Both seeds come from q and alpha in FP32, side by side.
// q within 2^+-60, alpha^2 <= q.  gamma is left as its seed and denominator
// (refine_gamma): nothing needs it before the next dot product is summed.
__device__ __forceinline__ void h7_scalars(double alpha, double q, double* sigma, double* seed, double* den) {
  const float qf = f32_of(q);
  const float rf = rsqrtf(qf);
  const float af = hi_abs(alpha) < ((1023 - 90) << 20) ? 0.0f : f32_of(fabs(alpha));
  const double g0 = f64_of(__fdividef(1.0f, fmaf(af, qf * rf, qf)));
  const double r = f64_of(rf);
  const double t = q * r;
  const double e = fma(-t, r, 1.0);
  const double te = t * e;
  const double p = fma(0.375, e, 0.5);
  const double sg = fma(te, p, t);
  *sigma = sg;
  *seed = g0;
  *den = fma(fabs(alpha), sg, q);
}

// 1 / den from its seed (one third-order step; seed exact when den = 1 / seed)
__device__ __forceinline__ double refine_gamma(double seed, double den) {
  const double e = fma(-den, seed, 1.0);
  return fma(seed, fma(e, e, e), seed);
}

// State of the critical warp between steps: reflector v, and its gamma as seed
// and denominator.
template <int R>
struct Crit {
  double v[R];
  double seed, den;
};

// One step of the critical warp: column j of S receives reflector j - 1 (kept
// from the last step) and becomes reflector j.  Lane l owns the rows l + 32 t.
// Leaf: head row j, tail rows j + 1 and on.  NODE: head row j of child 0, tail
// = the rows of the other children (zero below their diagonals).  Writes beta
// to row j, the unnormalised tail below it and the head to s_h[j].  gamma_(j-1)
// is refined here, beside the dot product, written to s_gam[j - 1] and
// announced on barrier kGamBar, where the column warps wait for it after their
// own dot products: the step barrier need not wait for it.
// Leaf: the block has `rows` rows, zero beyond them.
template <int R, bool NODE>
__device__ __forceinline__ void h7_crit(double* S, int ld, int j, Crit<R>& cr, double* s_h, double* s_gam,
                                        int nthreads, int rows) {
  const int lane = threadIdx.x & 31;
  double (&v)[R] = cr.v;
  double* col = S + (size_t)j * ld;
  double x[R];
#pragma unroll
  for (int t = 0; t < R; ++t) x[t] = col[lane + 32 * t];
  if (j > 0) {
    double d0 = v[0] * x[0], d1 = R > 1 ? v[1 % R] * x[1 % R] : 0.0;
    const double e = fma(-cr.den, cr.seed, 1.0);
#pragma unroll
    for (int t = 2; t < R; ++t) {
      if (t & 1) d1 = fma(v[t], x[t], d1);
      else d0 = fma(v[t], x[t], d0);
    }
    const double e2 = fma(e, e, e);
    if (R > 1) d0 += d1;
    const double gam = fma(cr.seed, e2, cr.seed);
    if (lane == 0) s_gam[j - 1] = gam;
    bar_arrive(kGamBar, nthreads);
    const double f = gam * warp_sum(d0);
#pragma unroll
    for (int t = 0; t < R; ++t) x[t] = fma(-f, v[t], x[t]);
  }
  const bool tail0 = !NODE && lane > j;
  const double y0 = (tail0 || lane == j) ? x[0] : 0.0;
  int nz = tail0 ? (hi_abs(x[0]) | __double2loint(x[0])) : 0;
#pragma unroll
  for (int t = 1; t < R; ++t) nz |= hi_abs(x[t]) | __double2loint(x[t]);
  double q = y0 * y0;
#pragma unroll
  for (int t = 1; t < R; ++t) q = fma(x[t], x[t], q);
  q = warp_sum(q);
  const double alpha = __shfl_sync(0xffffffffu, x[0], j);
  double h, beta;
  const int qh = __double2hiint(q);
  const bool usual = qh >= ((1023 - 60) << 20) && qh < ((1023 + 60) << 20);
  bool empty = !__any_sync(0xffffffffu, nz != 0);
  if (!NODE && !usual && !empty) {
    // a product 0 * NaN leaves NaN beyond the rows too; they are not part of the tail
    nz = 0;
#pragma unroll
    for (int t = 0; t < R; ++t) {
      const int r = lane + 32 * t;
      if (r >= rows) x[t] = 0.0;
      else if (r > j) nz |= hi_abs(x[t]) | __double2loint(x[t]);
    }
    empty = !__any_sync(0xffffffffu, nz != 0);
  }
  if (empty) {   // an empty tail: a sign flip
    h = 1.0;
    cr.seed = 2.0;
    cr.den = 0.5;
    beta = flip_if(alpha, true);
  } else {
    const bool neg = __double2hiint(alpha) < 0;
    if (usual) {
      double sigma;
      h7_scalars(alpha, q, &sigma, &cr.seed, &cr.den);
      h = alpha + flip_if(sigma, neg);
      beta = flip_if(sigma, !neg);
    } else {
      // squares outside the seeds' range: the reflector of the column scaled
      // by a power of two is the same reflector (v may carry any factor)
      int mx = (tail0 || lane == j) ? hi_abs(x[0]) : 0;
#pragma unroll
      for (int t = 1; t < R; ++t) mx = max(mx, hi_abs(x[t]));
      mx = __reduce_max_sync(0xffffffffu, (unsigned)mx);
      // Inf and NaN stay unscaled and spread as they would without the scaling
      const int e = mx >= 0x7ff00000 ? 0 : min(max((mx >> 20) - 1023, -1000), 1000);
      const double sc = __hiloint2double((1023 - e) << 20, 0), un = __hiloint2double((1023 + e) << 20, 0);
      if (tail0) x[0] *= sc;
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] *= sc;
      const double as = alpha * sc;
      const double z0 = lane == j ? as : (tail0 ? x[0] : 0.0);
      double qs = z0 * z0;
#pragma unroll
      for (int t = 1; t < R; ++t) qs = fma(x[t], x[t], qs);
      qs = warp_sum(qs);
      const double sigma = sqrt(qs);
      h = as + flip_if(sigma, neg);
      cr.den = fma(fabs(as), sigma, qs);
      cr.seed = 1.0 / cr.den;
      beta = flip_if(sigma, !neg) * un;
    }
  }
  col[lane] = lane == j ? beta : x[0];
#pragma unroll
  for (int t = 1; t < R; ++t) col[lane + 32 * t] = x[t];
  v[0] = lane == j ? h : (tail0 ? x[0] : 0.0);
#pragma unroll
  for (int t = 1; t < R; ++t) v[t] = x[t];
  if (lane == 0) s_h[j] = h;
}

// Reflector v with *gam applied to this warp's columns leaf_col(q, k0 + k), k <
// NC (*gam is there after barrier kGamBar).  The count is compiled in: an FP64
// instruction whose predicate is off for the whole warp still takes its slot.
template <int R, int NC>
__device__ __forceinline__ void h7_apply(double* S, int ld, int q, int k0, const double (&v)[R], const double* gam) {
  constexpr int N = NC <= 1 ? 1 : NC <= 2 ? 2 : NC <= 4 ? 4 : 8;
  constexpr bool keep = R <= 3;   // the columns stay in registers between their dot product and update
  const int lane = threadIdx.x & 31;
  double d[N];
  double xs[NC][keep ? R : 1];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    d[k] = 0.0;
    if (k < NC) {
      const double* sc = S + (size_t)leaf_col(q, k0 + k) * ld;
#pragma unroll
      for (int t = 0; t < R; ++t) {
        const double x = sc[lane + 32 * t];
        if constexpr (keep) xs[k < NC ? k : 0][t] = x;
        d[k] = fma(v[t], x, d[k]);
      }
    }
  }
  const double sum = warp_sum_held<N>(d);
  named_bar(kGamBar, kLeafStepThreads);
  const double f = *gam * sum;
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    const double fk = __shfl_sync(0xffffffffu, f, k * (32 / N));
    double* sc = S + (size_t)leaf_col(q, k0 + k) * ld;
    double x[R];
#pragma unroll
    for (int t = 0; t < R; ++t) {
      if constexpr (keep) x[t] = xs[k][t];
      else x[t] = sc[lane + 32 * t];
    }
#pragma unroll
    for (int t = 0; t < R; ++t) sc[lane + 32 * t] = fma(-fk, v[t], x[t]);
  }
}

struct NoPublish {
  __device__ void all(const double*, int, int, volatile int*, volatile int*) {}
};

// Householder QR of S (b columns, ld >= 32 R, rows beyond the data zero); all
// kLeafThreads threads call it after S is filled.  Afterwards S holds R (upper
// triangle) and the unnormalised tails, s_h the heads, s_gam the gammas.
// Step j: the critical warp finishes column j (see h7_crit) while the column
// warps apply reflector j - 1 to the columns after j; one barrier of those
// seven warps per step.  The publishing warp follows the count of finished
// columns on its own, so that its fences (about 1 us) hold nobody up.
template <int R, bool NODE, class Pub = NoPublish>
__device__ void h7_factor(double* S, int ld, int rows, int b, double* s_h, double* s_gam, volatile int* s_done,
                          Pub pub = Pub()) {
  const int lane = threadIdx.x & 31, warp = warp_id();
  const int q = bulk_index(warp);
  if (threadIdx.x == 0) *s_done = 0;
  __syncthreads();
  if (warp == 0 || q >= 0) {
    Crit<R> cr;
    double (&v)[R] = cr.v;
    const int kend = q >= 0 ? leaf_first(q, b) : 0;   // columns of this warp
    cr.seed = cr.den = 0.0;
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = 0.0;
    for (int j = 0; j < b; ++j) {
      named_bar(kStepBar, kLeafStepThreads);
      if (warp == 0) {
        h7_crit<R, NODE>(S, ld, j, cr, s_h, s_gam, kLeafStepThreads, rows);
        __threadfence_block();
        __syncwarp();
        if (lane == 0) *s_done = j + 1;
      } else if (j > 0) {
        const double* vj = S + (size_t)(j - 1) * ld;
        const double h = s_h[j - 1];
#pragma unroll
        for (int t = 0; t < R; ++t) v[t] = vj[lane + 32 * t];
        v[0] = lane == j - 1 ? h : (!NODE && lane > j - 1 ? v[0] : 0.0);
        const double* gam = s_gam + j - 1;
        // this warp's columns from j + 1 on are its last ones
        const int klo = leaf_first(q, j + 1);
        switch (kend - klo) {
          case 5: h7_apply<R, 5>(S, ld, q, klo, v, gam); break;
          case 4: h7_apply<R, 4>(S, ld, q, klo, v, gam); break;
          case 3: h7_apply<R, 3>(S, ld, q, klo, v, gam); break;
          case 2: h7_apply<R, 2>(S, ld, q, klo, v, gam); break;
          case 1: h7_apply<R, 1>(S, ld, q, klo, v, gam); break;
          default: named_bar(kGamBar, kLeafStepThreads); break;
        }
      }
    }
    if (warp == 0 && lane == 0) s_gam[b - 1] = refine_gamma(cr.seed, cr.den);
  } else if (warp == kPubWarp) {
    pub.all(S, ld, b, s_done, nullptr);
  }
  __syncthreads();
}

// Structure of an operand of mm32, on op(X).  The zeros (and unit diagonals)
// are stored; the structure only bounds the k range of a tile.
enum : int { kSDense = 0, kSUpper = 1, kSLower = 2 };

// C = C0 + alpha op(A) op(B) for b x b shared-memory blocks (b <= 32, zero
// beyond b up to whole 8 x 8 tiles; C0 may be nullptr, or C itself; C must not
// alias A or B), op(A)[i, k] = A[i ai + k ak], op(B)[k, j] = B[k bk + j bj].
// bo: rows and columns of C written, b, or up8(b) when C is an operand of a
// later product.  nb products with the same B at once: A and C advance by
// anext and cnext doubles.  All threads of the block call it.
// The 32 x 32 output is cut into 8 x 4 half tiles (lane l: row l % 8, column
// l / 8), one FP64 instruction per k, and a half tile's k loop covers only the
// structural nonzeros of its row and column blocks (empty for the zero tiles
// of a product of two upper-triangular operands).  They are dealt to eight
// warps (four in a block of four) in order of decreasing work, forward and
// backward in turn: two upper-triangular operands cost 88 FP64 instructions
// on the fullest sub-partition (80 on average).  One compact loop serves every
// product, because a call runs its code once: a version unrolled over the
// tiles waited for its instructions (7 us a product against 5).  Two sums per
// lane keep the FP64 pipe at its 65 cycles an instruction (76 in one chain).
__device__ __noinline__ void mm32(const double* A, int ai, int ak, int as, const double* B, int bk, int bj, int bs,
                                  double* C, int ldc, int bo, double alpha, const double* C0, int nb = 1,
                                  int anext = 0, int cnext = 0) {
  const int lane = threadIdx.x & 31, warp = warp_id();
  const int nw = blockDim.x >= 256 ? 8 : (int)blockDim.x >> 5;
  const int nt = (bo + 7) >> 3;
  int p = 0;
  for (int d = nt - 1; d > -nt; --d) {
    const int lo = d < 0 ? -d : 0, hi = d < 0 ? nt : nt - d;
    for (int t = lo * nb; t < hi * nb; ++t) {
      const int ti = nb == 1 ? t : t / nb, n = nb == 1 ? 0 : t - ti * nb;
#pragma unroll 1
      for (int half = 0; half < 2; ++half, ++p) {
        const int q = p & (2 * nw - 1);
        if ((q < nw ? q : 2 * nw - 1 - q) != warp) continue;
        const int i = 8 * ti + (lane & 7), j = 8 * (ti + d) + 4 * half + (lane >> 3);
        int k0 = 0, k1 = 8 * nt;
        if (as == kSUpper) k0 = 8 * ti;
        if (as == kSLower) k1 = min(k1, 8 * ti + 8);
        if (bs == kSUpper) k1 = min(k1, 8 * (ti + d) + 8);
        const double* pa = A + n * anext + i * ai + k0 * ak;
        const double* pb = B + j * bj + k0 * bk;
        double acc0 = 0.0, acc1 = 0.0;
#pragma unroll 1
        for (int k = k0; k < k1; k += 8) {
          double x[8], y[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            x[u] = pa[u * ak];
            y[u] = pb[u * bk];
          }
          pa += 8 * ak;
          pb += 8 * bk;
#pragma unroll
          for (int u = 0; u < 8; u += 2) {
            acc0 = fma(x[u], y[u], acc0);
            acc1 = fma(x[u + 1], y[u + 1], acc1);
          }
        }
        if (i < bo && j < bo)
          C[n * cnext + j * ldc + i] = fma(alpha, acc0 + acc1, C0 ? C0[j * ldc + i] : 0.0);
      }
    }
  }
  __syncthreads();
}

__device__ __forceinline__ int up8(int b) { return (b + 7) & ~7; }

// Inverse of the upper triangle of X (32 x 32, ld kLd) into Xi (ld kLd), by
// recursive 2 x 2 block inversion done bottom-up:
// inv([[A, B], [0, C]]) = [[A^-1, -A^-1 B C^-1], [0, C^-1]].  Every level is
// two small products computed in parallel, so the dependent FP64 chain is
// about 2 (1 + 2 + 4 + 8 + 16) operations instead of the b^2 / 2 of a
// substitution.  Only the leading w x w part (w = h4_width(b)) is read and written.
// scratch: 512 doubles.
__device__ __forceinline__ int h4_width(int b) { return b <= 8 ? 8 : b <= 16 ? 16 : kDirectB; }

template <int H>
__device__ __forceinline__ void h4_tri_level(const double* X, double* Xi, double* scratch, int width) {
  const int n = width / 2 * H;   // elements of the level's off-diagonal blocks
  constexpr int step = H < 8 ? H : 8;
  const int idx = threadIdx.x;
  const int p = idx / (H * H), e = idx % (H * H), i = e % H, j = e / H, i0 = p * 2 * H, c0 = i0 + H;
  double a0 = 0.0, a1 = 0.0;
  if (idx < n) {   // M = B C^-1 (C^-1 upper: zero below its diagonal)
#pragma unroll 1
    for (int k = 0; k <= j; k += step)
#pragma unroll
      for (int u = 0; u < step; ++u) {
        const double t = X[(c0 + k + u) * kLd + i0 + i], w = Xi[(c0 + j) * kLd + c0 + k + u];
        if (u & 1) a1 = fma(t, w, a1);
        else a0 = fma(t, w, a0);
      }
    scratch[idx] = a0 + a1;
  }
  __syncthreads();
  if (idx < n) {   // -A^-1 M
    a0 = a1 = 0.0;
#pragma unroll 1
    for (int k = i & ~(step - 1); k < H; k += step)
#pragma unroll
      for (int u = 0; u < step; ++u) {
        const double t = Xi[(i0 + k + u) * kLd + i0 + i], w = scratch[p * H * H + j * H + k + u];
        if (u & 1) a1 = fma(t, w, a1);
        else a0 = fma(t, w, a0);
      }
    Xi[(c0 + j) * kLd + i0 + i] = -(a0 + a1);
  }
  __syncthreads();
}

__device__ void h4_tri_inv(const double* X, int b, double* Xi, double* scratch) {
  const int width = h4_width(b);
  for (int idx = threadIdx.x; idx < width * kDirectB; idx += blockDim.x) {
    const int i = idx & 31, k = idx >> 5;
    if (i < width) Xi[k * kLd + i] = i == k ? quick_rcp(X[i * kLd + i]) : 0.0;
  }
  __syncthreads();
  h4_tri_level<1>(X, Xi, scratch, width);
  h4_tri_level<2>(X, Xi, scratch, width);
  h4_tri_level<4>(X, Xi, scratch, width);
  if (width > 8) h4_tri_level<8>(X, Xi, scratch, width);
  if (width > 16) h4_tri_level<16>(X, Xi, scratch, width);
}

// b x b block from global memory (ld b) into a shared block (ld kLd), zero beyond b
__device__ void h4_load(double* dst, const double* src, int b) {
  for (int idx = threadIdx.x; idx < kDirectB * kDirectB; idx += blockDim.x) {
    const int r = idx & 31, c = idx >> 5;
    dst[c * kLd + r] = (r < b && c < b) ? __ldcg(src + c * b + r) : 0.0;
  }
  __syncthreads();
}

// Rows [0, L) of b columns of a column-major block (ld lda) into S (ld ldS),
// zero up to row `rows` (a multiple of 32) and column h4_width(b): eight loads in
// flight per thread before any store.
__device__ void h4_load_block(double* S, int ldS, const double* A, int64_t lda, int L, int b, int rows) {
  const int n = rows * h4_width(b);
  for (int e0 = threadIdx.x; e0 < n; e0 += 8 * kLeafThreads) {
    double t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * kLeafThreads, c = e / rows, r = e - c * rows;
      t[u] = (r < L && c < b) ? A[(int64_t)c * lda + r] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * kLeafThreads, c = e / rows, r = e - c * rows;
      if (e < n) S[c * ldS + r] = t[u];
    }
  }
}

constexpr int kGramScratch = 4 * 640;   // h7_gram's partial sums (doubles)

// T^-1 = striu(V^T V) + diag(V^T V) / 2 of normalised reflectors into G (w x w,
// w = h4_width(b), ld kLd; columns beyond b get a unit diagonal).  V: rows 0..31 in
// VT (ld kLd, masked to the reflectors' structure), rows 32..rows-1 in S (ld ldS).
// Eight warps split the rows; each holds the upper 8 x 8 tiles (lane l: row l % 8
// of a tile, columns l / 8 and l / 8 + 4), so a row of 32 columns costs 20 FP64
// instructions and no shuffles; the eight partial sums meet in shared memory.
// NT = w / 8: with all ten tiles at every width, a 2000000 x 1 panel spent 3.3 ms in
// its leaves, most of it on columns that are not there.
template <int NT>
__device__ __forceinline__ void h7_gram_tiles(const double* VT, const double* S, int ldS, int rows, int b, double* G,
                                              double* part) {
  constexpr int TILES = NT * (NT + 1) / 2, PART = 64 * TILES;
  const int lane = threadIdx.x & 31, warp = warp_id();
  const int i = lane & 7, jj = lane >> 3;
  double acc[TILES][2];
#pragma unroll
  for (int t = 0; t < TILES; ++t) acc[t][0] = acc[t][1] = 0.0;
  if (warp < 8) {
    for (int r = warp; r < rows; r += 8) {
      const double* X = r < kDirectB ? VT : S;
      const int ld = r < kDirectB ? kLd : ldS;
      double x[NT], y0[NT], y1[NT];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        x[t] = X[(8 * t + i) * ld + r];
        y0[t] = X[(8 * t + jj) * ld + r];
        y1[t] = X[(8 * t + jj + 4) * ld + r];
      }
#pragma unroll
      for (int tj = 0; tj < NT; ++tj)
#pragma unroll
        for (int ti = 0; ti <= tj; ++ti) {
          const int t = tj * (tj + 1) / 2 + ti;
          acc[t][0] = fma(x[ti], y0[tj], acc[t][0]);
          acc[t][1] = fma(x[ti], y1[tj], acc[t][1]);
        }
    }
    if (warp >= 4) {
#pragma unroll
      for (int t = 0; t < TILES; ++t) {
        part[(warp - 4) * PART + t * 64 + lane] = acc[t][0];
        part[(warp - 4) * PART + t * 64 + 32 + lane] = acc[t][1];
      }
    }
  }
  __syncthreads();
  if (warp < 4) {
#pragma unroll
    for (int t = 0; t < TILES; ++t) {
      part[warp * PART + t * 64 + lane] += acc[t][0];
      part[warp * PART + t * 64 + 32 + lane] += acc[t][1];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < PART; e += blockDim.x) {
    const int t = e >> 6, u = (e >> 5) & 1, l = e & 31;
    int tj = 0;
    while ((tj + 1) * (tj + 2) / 2 <= t) ++tj;
    const int r = 8 * (t - tj * (tj + 1) / 2) + (l & 7), c = 8 * tj + (l >> 3) + 4 * u;
    const double g = (part[e] + part[PART + e]) + (part[2 * PART + e] + part[3 * PART + e]);
    if (r <= c) G[c * kLd + r] = r == c ? (c < b ? 0.5 * g : 1.0) : g;
  }
  __syncthreads();
}

__device__ void h7_gram(const double* VT, const double* S, int ldS, int rows, int b, double* G, double* part) {
  if (b <= 8) h7_gram_tiles<1>(VT, S, ldS, rows, b, G, part);
  else if (b <= 16) h7_gram_tiles<2>(VT, S, ldS, rows, b, G, part);
  else h7_gram_tiles<4>(VT, S, ldS, rows, b, G, part);
}

struct Hr4Args {
  double* A;
  int64_t lda;
  int64_t m;
  int b;
  double* Vw;       // m x b (ld m): leaf reflector vectors (strictly lower part; unit diagonal implied)
  double* Tl;       // P x b x b: leaf T factors
  double* Rn;       // nnodes x b x b: R of every node
  double* Qn;       // nnodes x kFan x b x b: node Q blocks
  unsigned* cnt;    // nnodes arrival counters (zeroed)
  double* T;        // out
  int64_t ldT;
  double* W;        // out or nullptr
  int64_t ldW;
  double* Uinv;     // scratch b x b
  int* status;
  unsigned* prog;   // pipelined tree: columns of R published by each node
  unsigned* done;   // pipelined tree: node finished (T, Q blocks, V written); the root's U^-1 last
  unsigned* ticket; // pipelined tree: role counter
  int* fail;        // pipelined tree: a wait gave up
  int polls, smem_polls;   // limits of the bounded waits
  double* Pc;       // pipelined tree: I - V0 T0 V0^T of leaf 0, then per level the product of the first
                    // Q blocks up leaf 0's path, (depth + 1) x b x b
  double* Mn;       // many leaves: per node, the product of the Q blocks from the root down to it
                    // times U^-1 (nnodes x b x b, by flat id), or nullptr
  int P;
  int yparts;       // pipelined tree: CTAs per leaf of k_hr6_y (0: k_hr4_form_y)
  int ldS;          // leading dimension of the shared block: 32 row slots + 1
  int depth;
  int nlev[kMaxLevels + 1];
  int base[kMaxLevels + 1];
};

__device__ __forceinline__ int h4_children(const Hr4Args& a, int lvl, int node) {
  // children of node (lvl, node) at level lvl-1
  const int first = node * kFan;
  const int n = a.nlev[lvl - 1] - first;
  return n < kFan ? n : kFan;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A wait ran out: the call's status, and in the pipelined tree the flag that ends the
// other CTAs' waits.
__device__ __forceinline__ void h6_give_up(int* fail, int* status) {
  if (fail) atomicExch(fail, 1);
  record_status(status, CANDMC_ERR_TIMEOUT);
}

constexpr int kBlk = kDirectB * kLd;        // doubles of a 32 x 32 shared block
constexpr int kRootDoubles = 6 * kBlk;

// The root: Q1_top, its sign-choice LU, T, W and U^-1.  The LU runs with a
// one-column lookahead: warp 0 applies column i to column i + 1 and finishes
// it (pivot, reciprocal, multipliers: a chain of six FP64 instructions) while
// three warps, with the columns in registers, apply column i to those beyond.
// U^-1 follows it column by column, X U = I giving X[:, c] = (e_c - sum_{k<c}
// X[:, k] U[k, c]) / U[c, c], by four warps that split the sum: Y waits for it.
// The same four then form T from T L^T = -U S, T[:, c] = -U[:, c] S_c -
// sum_{k<c} T[:, k] L[c, k], beside Y.  All loops are rolled: the role runs
// once on some SM, and unrolled over the columns it waits for its instructions
// (LU 32 us with eight columns a warp unrolled, 15 us rolled).  The LU, two
// inversions and a product one after the other took 58 us.
__device__ void h4_root(const Hr4Args& a, double* sm) {
  const int b = a.b, tid = threadIdx.x, lane = tid & 31, warp = warp_id();
  double* sR = sm;
  double* sL = sR + kBlk;    // Q1_top, becomes L\U
  double* sT = sL + kBlk;
  double* sX = sT + kBlk;    // U^-1
  double* sM = sX + kBlk;
  double* sQ = sM + kBlk;
  __shared__ int s_sign[kDirectB];
  __shared__ double s_rp[kDirectB], s_part[3][kDirectB];
  __shared__ volatile int s_cols, s_late;   // columns of L\U finished; a wait for one gave up
  for (int idx = tid; idx < kBlk; idx += blockDim.x) sQ[idx] = sL[idx] = 0.0;
  __syncthreads();
  if (a.Pc) {
    // the pipelined tree: sX (loaded by the caller) times the top node's first Q block
    if (a.depth > 0) {
      h4_load(sQ, a.Pc + (size_t)a.depth * b * b, b);
      mm32(sX, 1, kLd, kSDense, sQ, 1, kLd, kSUpper, sL, kLd, up8(b), 1.0, nullptr);
    } else {
      h4_load(sL, a.Pc, b);
    }
  } else {
    // chain M = Q1^(1) ... Q1^(depth) of the first-child Q blocks (upper triangular)
    for (int idx = tid; idx < kBlk; idx += blockDim.x) {
      const int r = idx % kLd, c = idx / kLd;
      sM[idx] = (r == c && c < b) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int lvl = a.depth; lvl >= 1; --lvl) {
      if (h4_children(a, lvl, 0) > 1) {
        h4_load(sX, a.Qn + ((size_t)a.base[lvl] * kFan + 0) * b * b, b);
        mm32(sX, 1, kLd, kSUpper, sM, 1, kLd, kSUpper, sQ, kLd, up8(b), 1.0, nullptr);
        for (int idx = tid; idx < b * b; idx += blockDim.x) sM[(idx / b) * kLd + idx % b] = sQ[(idx / b) * kLd + idx % b];
        __syncthreads();
      }
    }
    // Q1_top = C0 - V0 (T0 (V0^T C0)), V0 = unit-lower top block of leaf 0, C0 = M
    for (int idx = tid; idx < kBlk; idx += blockDim.x) {
      const int r = idx % kLd, c = idx / kLd;
      sL[idx] = (r < b && c < b) ? (r > c ? __ldcg(a.Vw + (int64_t)c * a.m + r) : (r == c ? 1.0 : 0.0)) : 0.0;
    }
    h4_load(sT, a.Tl, b);
    mm32(sL, kLd, 1, kSUpper, sM, 1, kLd, kSUpper, sX, kLd, up8(b), 1.0, nullptr);    // V0^T C0 (upper)
    mm32(sT, 1, kLd, kSUpper, sX, 1, kLd, kSUpper, sQ, kLd, up8(b), 1.0, nullptr);   // T0 of it (upper)
    mm32(sL, 1, kLd, kSLower, sQ, 1, kLd, kSUpper, sX, kLd, up8(b), -1.0, sM);       // C0 - V0 sQ
    for (int idx = tid; idx < b * b; idx += blockDim.x) sL[(idx / b) * kLd + idx % b] = sX[(idx / b) * kLd + idx % b];
    __syncthreads();
  }
  for (int idx = tid; idx < kBlk; idx += blockDim.x) sT[idx] = sX[idx] = 0.0;
  if (tid == 0) s_cols = s_late = 0;
  __syncthreads();
  // columns before c finished (one warp)
  auto wait_cols = [&](int c) {
    int it = 0;
    while (s_cols < c && ++it < a.smem_polls) __nanosleep(it < 1024 ? 20 : 100);
    __syncwarp();
    if (lane == 0 && it >= a.smem_polls) {
      h6_give_up(a.fail, a.status);
      s_late = 1;
    }
    __threadfence_block();
  };
  // acc minus the sum over k < c, k = h (mod 4), of X[:, k] v[k], four terms at a
  // time (those from c on read as zero)
  const int h = warp - 1;   // of the four warps 1..4
  auto minus_sum = [&](double acc, const double* X, const double* v, int ldv, int c) -> double {
#pragma unroll 1
    for (int k = h; k < c; k += 16) {
      double x[4], u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int kk = k + 4 * q;
        x[q] = kk < c ? X[kk * kLd + lane] : 0.0;
        u[q] = kk < c ? v[kk * ldv] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) acc = fma(-x[q], u[q], acc);
    }
    return acc;
  };
  if (warp == 0) {
    double x = sL[lane];
    for (int i = 0; i < b; ++i) {
      const double d = __shfl_sync(0xffffffffu, x, i);
      const long long db = __double_as_longlong(d);
      const bool pos = db > 0 && db <= 0x7ff0000000000000LL;   // d > 0
      // 1 <= |piv| <= 2: the sign choice keeps the pivot away from 0 (a NaN
      // passes through the refinement below)
      const double piv = d + (pos ? 1.0 : -1.0);
      const double y = flip_if(f64_of(__fdividef(1.0f, f32_of(fabs(piv)))), !pos);
      const double e = fma(-piv, y, 1.0);
      const double xy = x * y;
      const double e2 = fma(e, e, e);
      const double m = fma(xy, e2, xy);   // the multipliers x / piv
      sL[i * kLd + lane] = lane > i ? m : (lane == i ? piv : x);
      if (lane == 0) {
        s_sign[i] = pos ? -1 : 1;
        s_rp[i] = fma(y, e2, y);
      }
      __threadfence_block();
      __syncwarp();
      if (lane == 0) s_cols = i + 1;
      named_bar(1, 4 * 32);
      if (i + 1 < b) {
        const double xn = sL[(i + 1) * kLd + lane];
        const double u = __shfl_sync(0xffffffffu, xn, i);
        x = lane > i ? fma(-m, u, xn) : xn;
      }
    }
  } else if (warp >= 5 && warp <= 7) {
    // columns q, q + 3, .. in registers (one row per lane); column i + 2 goes
    // back to shared memory for the critical warp when it is next
    const int q = warp - 5;
    double x[11];
#pragma unroll
    for (int k = 0; k < 11; ++k) {
      const int c = q + 3 * k;
      x[k] = c < kDirectB ? sL[c * kLd + lane] : 0.0;
    }
#pragma unroll 1
    for (int i = 0; i < b; ++i) {
      named_bar(1, 4 * 32);
      const double l = lane > i ? sL[i * kLd + lane] : 0.0;
#pragma unroll
      for (int k = 10; k >= 0; --k) {   // a break, not a predicate: see h7_apply
        const int c = q + 3 * k;
        if (c < i + 2) break;
        if (c < kDirectB) x[k] = fma(-l, __shfl_sync(0xffffffffu, x[k], i), x[k]);
        if (c == i + 2) sL[c * kLd + lane] = x[k];
      }
    }
  } else if (warp <= 4) {
    bool bad = false;
#pragma unroll 1
    for (int c = 0; c < b; ++c) {
      wait_cols(c + 1);
      const double acc = minus_sum((h == 0 && lane == c) ? 1.0 : 0.0, sX, sL + c * kLd, 1, c);
      if (h) s_part[h - 1][lane] = acc;
      named_bar(2, 128);
      if (!h) {
        const double v =
            lane <= c ? ((acc + s_part[0][lane]) + (s_part[1][lane] + s_part[2][lane])) * s_rp[c] : 0.0;
        sX[c * kLd + lane] = v;
        if (lane < b) a.Uinv[c * b + lane] = v;
        bad |= hi_abs(v) >= 0x7ff00000;
      }
      named_bar(2, 128);
    }
    if (!h) {
      if (bad) record_status(a.status, CANDMC_ERR_NUMERIC);
      __threadfence();
      __syncwarp();
      if (lane == 0 && a.Pc && !s_late) st_release(a.done + a.base[a.depth] + 1, 1u);
    }
#pragma unroll 1
    for (int c = 0; c < b; ++c) {
      const double acc = minus_sum((h == 0 && lane <= c) ? flip_if(sL[c * kLd + lane], s_sign[c] > 0) : 0.0, sT,
                                   sL + c, kLd, c);
      if (h) s_part[h - 1][lane] = acc;
      named_bar(2, 128);
      if (!h)
        sT[c * kLd + lane] = lane <= c ? (acc + s_part[0][lane]) + (s_part[1][lane] + s_part[2][lane]) : 0.0;
      named_bar(2, 128);
    }
  } else if (warp == 8) {   // R while the others work
    for (int c = 0; c < b; ++c)
      if (lane < b) sR[c * kLd + lane] = __ldcg(a.Rn + (size_t)a.base[a.depth] * b * b + c * b + lane);
  }
  __syncthreads();
  for (int idx = tid; idx < b * b; idx += blockDim.x) {
    const int r = idx % b, c = idx / b;
    const double lu = sL[c * kLd + r];
    a.A[c * a.lda + r] = (r > c) ? lu : flip_if(sR[c * kLd + r], s_sign[r] < 0);
    if (a.W) a.W[c * a.ldW + r] = (r <= c) ? flip_if(lu, s_sign[c] < 0) : 0.0;
    a.T[c * a.ldT + r] = (r <= c) ? sT[c * kLd + r] : 0.0;
  }
}

// The reflectors of a factored leaf: S's tails divided by their heads (s_h
// becomes the reciprocals), written to Vw (strictly lower part, L rows), and
// the masked top 32 rows in VT.
__device__ void h7_leaf_v(double* S, int ldS, int L, int rows, int b, double* s_h, double* VT, double* Vw, int64_t m) {
  const int tid = threadIdx.x;
  if (tid < kDirectB) s_h[tid] = tid < b ? quick_rcp(s_h[tid]) : 0.0;
  __syncthreads();
  const int n = rows * h4_width(b);
  for (int e = tid; e < n; e += kLeafThreads) {
    const int c = e / rows, r = e - c * rows;
    double v = 0.0;
    if (r > c && c < b) {
      v = S[c * ldS + r] * s_h[c];
      S[c * ldS + r] = v;
    }
    if (r < kDirectB) VT[c * kLd + r] = (r == c && c < b) ? 1.0 : v;
    if (r < L && c < b) Vw[(int64_t)c * m + r] = v;
  }
  __syncthreads();
}

__device__ __forceinline__ int h7_slots(int L) {
  const int s = (L + 31) >> 5;
  return s <= 4 ? s : kMaxR;
}

template <class Pub>
__device__ void h7_leaf_factor(double* S, int ldS, int slots, int L, int b, double* s_h, double* s_gam, Pub pub) {
  __shared__ volatile int s_done;
  switch (slots) {
    case 1: h7_factor<1, false>(S, ldS, L, b, s_h, s_gam, &s_done, pub); break;
    case 2: h7_factor<2, false>(S, ldS, L, b, s_h, s_gam, &s_done, pub); break;
    case 3: h7_factor<3, false>(S, ldS, L, b, s_h, s_gam, &s_done, pub); break;
    case 4: h7_factor<4, false>(S, ldS, L, b, s_h, s_gam, &s_done, pub); break;
    default: h7_factor<kMaxR, false>(S, ldS, L, b, s_h, s_gam, &s_done, pub); break;
  }
}

// shared memory of a leaf after its block S: VT, G, and the scratch that holds
// h7_gram's partial sums, then h4_tri_inv's products and T
constexpr int kLeafScratch = kGramScratch > 512 + kBlk ? kGramScratch : 512 + kBlk;

__global__ void __launch_bounds__(kLeafThreads, 2) k_hr4_leaf_tree(Hr4Args a) {
  extern __shared__ double sm4[];
  __shared__ double s_h[kDirectB], s_gam[kDirectB];
  __shared__ int s_last;
  __shared__ volatile int s_done;
  const int b = a.b, tid = threadIdx.x;
  const int leaf = blockIdx.x;
  const int64_t r0 = t4_leaf_row0(a.m, a.P, leaf);
  const int L = (int)(t4_leaf_row0(a.m, a.P, leaf + 1) - r0);
  const int ldS = a.ldS;
  double* S = sm4;
  double* VT = S + (size_t)ldS * kDirectB;
  double* G = VT + kBlk;
  double* scratch = G + kBlk;
  double* Tt = scratch + 512;

  // ---- leaf: Householder QR of rows [r0, r0 + L); the rows beyond L are zero
  const int slots = h7_slots(L);
  h4_load_block(S, ldS, a.A + r0, a.lda, L, b, 32 * slots);
  h7_leaf_factor(S, ldS, slots, L, b, s_h, s_gam, NoPublish());
  double* Rl = a.Rn + (size_t)(a.base[0] + leaf) * b * b;
  for (int idx = tid; idx < b * b; idx += blockDim.x) {
    const int r = idx % b, c = idx / b;
    Rl[idx] = (r <= c) ? S[c * ldS + r] : 0.0;
  }
  h7_leaf_v(S, ldS, L, 32 * slots, b, s_h, VT, a.Vw + r0, a.m);
  h7_gram(VT, S, ldS, 32 * slots, b, G, scratch);
  h4_tri_inv(G, b, Tt, scratch);
  double* Tleaf = a.Tl + (size_t)leaf * b * b;
  for (int idx = tid; idx < b * b; idx += blockDim.x) Tleaf[idx] = (idx % b <= idx / b) ? Tt[(idx / b) * kLd + idx % b] : 0.0;

  // ---- climb the fan-in-4 tree
  int node = leaf;
  for (int lvl = 0; lvl < a.depth; ++lvl) {
    const int parent = node / kFan;
    const int nch = h4_children(a, lvl + 1, parent);
    double* Rpar = a.Rn + (size_t)(a.base[lvl + 1] + parent) * b * b;
    if (nch == 1) {
      const double* Rme = a.Rn + (size_t)(a.base[lvl] + node) * b * b;
      __syncthreads();
      for (int idx = tid; idx < b * b; idx += blockDim.x) Rpar[idx] = __ldcg(Rme + idx);
      __syncthreads();
      node = parent;
      continue;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = (atomicAdd(a.cnt + a.base[lvl + 1] + parent, 1u) == (unsigned)(nch - 1));
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // stack the children's R factors: child k occupies rows [32 k, 32 k + b)
    // (rows b..31 of every child, and the children beyond nch, stay zero)
    for (int idx = tid; idx < h4_width(b) * kFan * 32; idx += blockDim.x) {
      const int c = idx / (kFan * 32), r = idx % (kFan * 32), k = r >> 5, i = r & 31;
      const double* Rk = a.Rn + (size_t)(a.base[lvl] + parent * kFan + k) * b * b;
      S[c * ldS + r] = (k < nch && c < b && i <= c) ? __ldcg(Rk + c * b + i) : 0.0;
    }
    // reflector j: head row j (child 0), tail = rows 0..j of every other child
    // (the children are upper triangular, so nothing below their diagonals is touched)
    h7_factor<kFan, true>(S, ldS, kFan * 32, b, s_h, s_gam, &s_done);
    for (int idx = tid; idx < b * b; idx += blockDim.x) {
      const int r = idx % b, c = idx / b;
      Rpar[idx] = (r <= c) ? S[c * ldS + r] : 0.0;
    }
    // V = [I; V_1; ..; V_{nch-1}] (V_k upper triangular), normalised
    if (tid < kDirectB) s_h[tid] = tid < b ? quick_rcp(s_h[tid]) : 0.0;
    __syncthreads();
    for (int idx = tid; idx < h4_width(b) * kFan * 32; idx += blockDim.x) {
      const int c = idx / (kFan * 32), r = idx % (kFan * 32);
      if (r >= 32) S[c * ldS + r] *= s_h[c];
      else VT[c * kLd + r] = (r == c && c < b) ? 1.0 : 0.0;
    }
    __syncthreads();
    h7_gram(VT, S, ldS, kFan * 32, b, G, scratch);
    h4_tri_inv(G, b, Tt, scratch);
    double* Qp = a.Qn + (size_t)(a.base[lvl + 1] + parent) * kFan * b * b;
    // Q_1 = I - T;  Q_k = -V_k T
    for (int idx = tid; idx < b * b; idx += blockDim.x) {
      const int r = idx % b, c = idx / b;
      Qp[idx] = ((r == c) ? 1.0 : 0.0) - ((r <= c) ? Tt[c * kLd + r] : 0.0);
    }
    for (int k = 1; k < nch; ++k) {
      double* Qk = G;   // G is free once T is formed
      mm32(S + 32 * k, 1, ldS, kSUpper, Tt, 1, kLd, kSUpper, Qk, kLd, b, -1.0, nullptr);
      for (int idx = tid; idx < b * b; idx += blockDim.x) Qp[(size_t)k * b * b + idx] = Qk[(idx / b) * kLd + idx % b];
      __syncthreads();
    }
    node = parent;
  }
  __threadfence();
  __syncthreads();
  h4_root(a, sm4);
}

// ---- pipelined tree: one launch for the leaves and every internal node.
//
// The levels of the tree above do not overlap: a node starts when its
// children have finished all b columns, so a panel costs (1 + depth) b
// sequential Householder steps.  Here a node starts column j as soon as its
// children have published column j of their R: leaves run the right-looking
// steps above and publish each column of R when it becomes final; internal
// nodes run left-looking, applying their earlier reflectors to the arriving
// column through the compact-WY factor T they build as they go (LAPACK
// dlarft's column recurrence T[0:j, j] = -tau_j T[0:j, 0:j] V^T v_j), so the
// panel costs about b + depth steps.  Roles come from an atomic ticket
// (leaves first, then the nodes level by level), so a node only waits for
// CTAs that took a lower ticket and are already running, whatever the
// scheduling order.  Every wait is bounded: a wait that runs out, on another CTA
// or on a warp of its own, records CANDMC_ERR_TIMEOUT and sets the flag that every
// wait on another CTA polls, and the CTA returns without publishing anything more,
// so no other CTA is left waiting on it or takes what it did not finish.

// One thread: wait until *p >= v.  False when the wait gave up or another CTA
// of this launch did.
__device__ bool h6_wait(const Hr4Args& a, const unsigned* p, unsigned v) {
  for (int it = 0; it < a.polls; ++it) {
    if (ld_acquire(p) >= v) return true;
    if (*(volatile int*)a.fail) return false;
    if (it > 8) __nanosleep(100);
  }
  h6_give_up(a.fail, a.status);
  return false;
}

// R handed to the parent column by column (rows 0..j of S's column j) as the
// count *s_done of finished columns grows, by one warp.  Stops when *s_fail
// (may be nullptr) is set; where its own wait runs out it sets *s_short (apart
// from s_fail, which the column warps read between their barriers).
struct Publish {
  double* Rcol;
  int b;
  unsigned* prog;
  volatile int* s_short;
  int polls;
  int *fail, *status;
  __device__ void all(const double* S, int ld, int n, volatile int* s_done, volatile int* s_fail) {
    const int lane = threadIdx.x & 31;
    for (int j = 0; j < n; ++j) {
      for (int it = 0; *s_done <= j && !(s_fail && *s_fail);) {
        if (++it >= polls) break;
        __nanosleep(it < 1024 ? 20 : 100);
      }
      if (__any_sync(0xffffffffu, *s_done <= j)) {
        if (lane == 0 && !(s_fail && *s_fail)) {
          h6_give_up(fail, status);
          *s_short = 1;
        }
        return;
      }
      __threadfence_block();
      if (lane <= j) Rcol[j * b + lane] = S[j * ld + lane];
      __syncwarp();   // orders the lanes' stores before lane 0's release
      if (lane == 0) st_release(prog, (unsigned)(j + 1));
    }
  }
};

__device__ void h6_leaf(const Hr4Args& a, int leaf, double* sm, double* s_h, double* s_gam) {
  __shared__ volatile int s_short;
  const int b = a.b, tid = threadIdx.x;
  const int64_t r0 = t4_leaf_row0(a.m, a.P, leaf);
  const int L = (int)(t4_leaf_row0(a.m, a.P, leaf + 1) - r0);
  const int ldS = a.ldS;
  double* S = sm;
  double* VT = S + (size_t)ldS * kDirectB;
  double* G = VT + kBlk;
  double* scratch = G + kBlk;
  double* Tt = scratch + 512;
  const int slots = h7_slots(L);
  if (tid == 0) s_short = 0;   // read after the barriers of the factorization
  h4_load_block(S, ldS, a.A + r0, a.lda, L, b, 32 * slots);
  h7_leaf_factor(S, ldS, slots, L, b, s_h, s_gam,
                 Publish{a.Rn + (size_t)leaf * b * b, b, a.prog + leaf, &s_short, a.smem_polls, a.fail, a.status});
  if (s_short) return;
  h7_leaf_v(S, ldS, L, 32 * slots, b, s_h, VT, a.Vw + r0, a.m);
  h7_gram(VT, S, ldS, 32 * slots, b, G, scratch);
  h4_tri_inv(G, b, Tt, scratch);
  double* Tleaf = a.Tl + (size_t)leaf * b * b;
  for (int idx = tid; idx < b * b; idx += blockDim.x) Tleaf[idx] = (idx % b <= idx / b) ? Tt[(idx / b) * kLd + idx % b] : 0.0;
  if (leaf == 0 && a.Pc) {
    // P_0 = I - V0 T0 V0^T on the top b rows (V0 unit lower): the first factor
    // of Q1_top, multiplied by the path nodes' Q1 blocks as they finish
    mm32(Tt, 1, kLd, kSUpper, VT, kLd, 1, kSUpper, G, kLd, up8(b), 1.0, nullptr);   // G = T0 V0^T
    mm32(VT, 1, kLd, kSLower, G, 1, kLd, kSUpper, S, kLd, b, 1.0, nullptr);        // V0 G (S is free)
    for (int idx = tid; idx < b * b; idx += blockDim.x)
      a.Pc[idx] = ((idx % b == idx / b) ? 1.0 : 0.0) - S[(idx / b) * kLd + idx % b];
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    if (leaf == 0) st_release(a.prog + 0, (unsigned)b + 1u);
    st_release(a.done + leaf, 1u);
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr int kNodeLd = kFan * 32 + 1;   // child k at rows [32 k, 32 k + b)
constexpr int kNodeDoubles = kNodeLd * kDirectB + 4 * kBlk + 4 * 96 + 2 * 32;

// One warp's triangular matrix-vector product: lane l < n returns the sum over
// t <= l of x(l, t) y(l, t).  Row l has l + 1 terms, so rows l and n - 1 - l
// together have n + 1: the longer one keeps its first h = (n + 2) / 2 terms and
// the lane of the shorter one takes the rest after its own, which halves the
// FP64 instructions of a loop over t <= l with idle lanes (17 instead of 31 at
// n = 31).  Terms outside load as zero: a divergent branch per term cost more
// than the fma (150 cycles a term instead of 76).
template <class X, class Y>
__device__ __forceinline__ double tri_fold(int n, X x, Y y) {
  const int lane = threadIdx.x & 31;
  const int mirror = n - 1 - lane, h = (n + 2) >> 1;
  const bool big = 2 * lane > n - 1;
  const int sw = (big || lane + 1 >= h) ? 64 : lane + 1;   // from here on the lane helps row `mirror`
  double acc = 0.0, own = 0.0;
  for (int t0 = 0; t0 < h; t0 += 4) {
    double xv[4], yv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = t0 + u;
      const int l = t >= sw ? mirror : lane, q = t >= sw ? h + t - sw : t;
      const bool in = t < h && lane < n && q <= l;
      xv[u] = in ? x(l, q) : 0.0;
      yv[u] = in ? y(l, q) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (t0 + u == sw) {
        own = acc;
        acc = 0.0;
      }
      acc = fma(xv[u], yv[u], acc);
    }
  }
  const bool helped = sw < 64;
  const double rest = __shfl_sync(0xffffffffu, helped ? acc : 0.0, mirror & 31);
  return big ? acc + rest : (helped ? own : acc);
}

// An internal node.  V = [D; V_1; V_2; V_3] with the reflectors unnormalised
// (D = diag(h)) and T of that form (T_pp = gamma_p).  Step j, between two
// barriers of the critical and the column warps:
//  * warp 0 applies reflector j - 1 to column j and forms reflector j;
//  * warps 1-3, one per child, apply the reflectors before j to column j + 1:
//    z = V^T s with one reflector per lane (no reduction over lanes), w = T^T z
//    with the columns of T the last step knew, s -= V w with one row per lane;
//  * warps 5-7, one per child, form column j - 1 of T: y = V^T v_(j-1),
//    T[0:j-1, j-1] = -gamma_(j-1) T y, and the last entry of w, gamma_(j-1)
//    (z_(j-1) - (T y)^T z), while warps 1-3 apply the others;
//  * the polling warp fetches the children's columns as they appear, and the
//    publishing warp hands finished columns to the parent, both at their own
//    pace (a fence or a trip to L2 takes about as long as a short step).
// V_k is upper triangular, so z, y and V w run folded (tri_fold).
// Bound: the FP64 pipes of the three sub-partitions with the column warps,
// about 92 instructions a step at j = 31 and half that on average (131 with
// the triangles unfolded: 122 us for 32 columns whose leaves take 79).
__device__ void h6_node(const Hr4Args& a, int f, double* sm, double* s_h, double* s_gam) {
  const int b = a.b, tid = threadIdx.x, lane = tid & 31, warp = warp_id();
  __shared__ int s_okv[2];
  __shared__ volatile int s_done, s_got, s_fail;   // columns finished, fetched; a wait for a column gave up
  __shared__ volatile int s_short;                 // the publishing warp's gave up
  int lvl = 1;
  while (lvl < a.depth && f >= a.base[lvl + 1]) ++lvl;
  const int idx = f - a.base[lvl];
  const int nch = h4_children(a, lvl, idx);
  const int child0 = a.base[lvl - 1] + idx * kFan;   // flat id of child 0
  double* Rme = a.Rn + (size_t)f * b * b;
  constexpr int ld = kNodeLd;
  double* S = sm;
  double* Tn = S + ld * kDirectB;
  double* Qk = Tn + kBlk;
  double* Pb = Qk + kBlk;
  double* Po = Pb + kBlk;
  double* zp = Po + kBlk;     // 3 x 32 partial sums each
  double* yp = zp + 96;
  double* wp = yp + 96;
  double* tp = wp + 96;
  double* zs = tp + 96;       // z, and w of the last reflector
  double* wl = zs + 32;
  if (nch == 1) {   // a pass-through node: its R is its child's
    if (warp == 0) {
      bool ok = true;
      for (int j = 0; ok && j < b; ++j) {
        if (lane == 0) ok = h6_wait(a, a.prog + child0, (unsigned)(j + 1));
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        if (!ok) break;
        if (lane <= j) Rme[j * b + lane] = __ldcg(a.Rn + (size_t)child0 * b * b + j * b + lane);
        __threadfence();
        __syncwarp();
        if (lane == 0) st_release(a.prog + f, (unsigned)(j + 1));
      }
      if (lane == 0) s_okv[0] = ok;
    }
    __syncthreads();
    if (!s_okv[0]) return;
  } else {
    for (int i = tid; i < ld * kDirectB; i += blockDim.x) S[i] = 0.0;
    for (int i = tid; i < kBlk; i += blockDim.x) Tn[i] = 0.0;
    if (tid == 0) s_done = s_got = s_fail = s_short = 0;
    __syncthreads();
    Publish pub{Rme, b, a.prog + f, &s_short, a.smem_polls, a.fail, a.status};
    // column c of the children's R into S (polling warp: lane k waits for child k)
    auto fetch = [&](int c) -> bool {
      bool ok = true;
      if (lane < nch) ok = h6_wait(a, a.prog + child0 + lane, (unsigned)(c + 1));
      if (!__all_sync(0xffffffffu, ok)) return false;
      double t[kFan];
#pragma unroll
      for (int k = 0; k < kFan; ++k)
        t[k] = (k < nch && lane <= c) ? __ldcg(a.Rn + (size_t)(child0 + k) * b * b + c * b + lane) : 0.0;
#pragma unroll
      for (int k = 0; k < kFan; ++k) S[c * ld + 32 * k + lane] = t[k];
      return true;
    };
    const int kc = warp & 3;                 // the child of a column warp: 1..3
    const bool tgrp = warp >= 5 && warp <= 7;
    const bool cgrp = warp >= 1 && warp <= 3;
    // reflectors 0..n-1 are formed: column n - 1 of T, and the reflectors
    // applied to column c (when c < b)
    auto bulk = [&](int n, int c) {
      const double* Vk = S + 32 * kc;
      const bool live = kc < nch;
      double acc = 0.0;
      if (tgrp) {
        if (live)
          acc = tri_fold(n - 1, [&](int p, int r) { return Vk[p * ld + r]; }, [&](int, int r) { return Vk[(n - 1) * ld + r]; });
        yp[(kc - 1) * 32 + lane] = acc;
      } else {
        if (live && c < b)
          acc = tri_fold(n, [&](int p, int r) { return Vk[p * ld + r]; }, [&](int, int r) { return Vk[c * ld + r]; });
        zp[(kc - 1) * 32 + lane] = acc;
      }
      named_bar(1, kBulkWarps * 32);
      // the sums over the children; then this warp's third of T y or T^T z
      // (columns beyond what is known are zero in Tn)
      double z = 0.0;
      acc = 0.0;
      if (tgrp) {
        const double y = (yp[lane] + yp[32 + lane]) + yp[64 + lane];
        for (int q = kc - 1; q < n - 1; q += 12) {
          double t[4], w[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = q + 3 * u;
            t[u] = k < n - 1 ? Tn[k * kLd + lane] : 0.0;
            w[u] = __shfl_sync(0xffffffffu, y, k & 31);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (q + 3 * u < n - 1) acc = fma(t[u], w[u], acc);
        }
        tp[(kc - 1) * 32 + lane] = acc;
      } else if (c < b) {
        if (lane < n) z = fma(s_h[lane], S[c * ld + lane], (zp[lane] + zp[32 + lane]) + zp[64 + lane]);
        if (kc == 1) zs[lane] = z;
        for (int q = kc - 1; q < n - 1; q += 12) {
          double t[4], w[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = q + 3 * u;
            t[u] = (k < n - 1 && lane < n - 1) ? Tn[lane * kLd + k] : 0.0;
            w[u] = __shfl_sync(0xffffffffu, z, k & 31);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (q + 3 * u < n - 1) acc = fma(t[u], w[u], acc);
        }
        wp[(kc - 1) * 32 + lane] = acc;
      }
      named_bar(1, kBulkWarps * 32);
      if (n < b) named_bar(kGamBar, kStepThreads);
      if (tgrp) {
        const double g = s_gam[n - 1];
        const double t = (tp[lane] + tp[32 + lane]) + tp[64 + lane];
        if (kc == 1) {
          if (lane < n) Tn[(n - 1) * kLd + lane] = lane < n - 1 ? -g * t : g;
        } else if (kc == 2 && c < b) {
          // w_(n-1) = gamma (z_(n-1) - (T y)^T z), while warps 1-3 work on the rest
          const double u = warp_sum(lane < n - 1 ? t * zs[lane] : 0.0);
          if (lane == 0) *wl = g * (zs[n - 1] - u);
          named_bar(2, 4 * 32);
        }
      } else if (c < b) {
        // s -= V w: row r = n - 2 - l takes the reflectors p = n - 2 - t >= r,
        // then reflector n - 1 everywhere
        const double w = lane < n - 1 ? (wp[lane] + wp[32 + lane]) + wp[64 + lane] : 0.0;
        double* ws = zp + (kc - 1) * 32;   // the partial z of this warp's child is done
        ws[lane] = w;
        __syncwarp();
        acc = tri_fold(n - 1, [&](int l, int t) { return Vk[(n - 2 - t) * ld + n - 2 - l]; },
                       [&](int, int t) { return ws[n - 2 - t]; });
        // to row order: lane l has row n - 2 - l
        acc = __shfl_sync(0xffffffffu, acc, (n - 2 - lane) & 31);
        if (lane >= n - 1) acc = 0.0;
        named_bar(2, 4 * 32);
        const double wn = *wl;
        if (live && lane < n) S[c * ld + 32 * kc + lane] -= fma(Vk[(n - 1) * ld + lane], wn, acc);
        if (kc == 1 && lane < n) S[c * ld + lane] = fma(-s_h[lane], lane == n - 1 ? wn : w, S[c * ld + lane]);
      }
    };
    if (warp == 0 || tgrp || cgrp) {
      Crit<kFan> cr;
      cr.seed = cr.den = 0.0;
#pragma unroll
      for (int t = 0; t < kFan; ++t) cr.v[t] = 0.0;
      for (int j = 0; j < b; ++j) {
        if (warp == 0) {
          // columns up to j + 1 must have arrived (the polling warp's own wait is as
          // long, and sets s_fail)
          const int need = j + 2 < b ? j + 2 : b;
          int it = 0, polls = a.smem_polls;
          while (s_got < need && !s_fail && ++it < polls)
            if (it >= 4096) __nanosleep(100);
          __syncwarp();
          if (lane == 0 && it >= polls) h6_give_up(a.fail, a.status);
          if (lane == 0) s_okv[j & 1] = s_got >= need;
          __threadfence_block();
        }
        named_bar(kStepBar, kStepThreads);
        if (!s_okv[j & 1]) {   // written before this barrier, rewritten two barriers on
          s_fail = 1;
          break;
        }
        if (warp == 0) {
          h7_crit<kFan, true>(S, ld, j, cr, s_h, s_gam, kStepThreads, 0);
          __threadfence_block();
          __syncwarp();
          if (lane == 0) s_done = j + 1;
        } else if (j > 0) {
          bulk(j, j + 1);
        }
      }
      if (warp == 0 && lane == 0) s_gam[b - 1] = refine_gamma(cr.seed, cr.den);
      named_bar(kStepBar, kStepThreads);
      if (warp != 0 && !s_fail) bulk(b, b);
    } else if (warp == kPollWarp) {
      for (int c = 0; c < b; ++c) {
        if (!fetch(c)) {
          s_fail = 1;
          break;
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0) s_got = c + 1;
      }
    } else {
      pub.all(S, ld, b, &s_done, &s_fail);
    }
    __syncthreads();
    if (s_fail || s_short) return;
    // T of normalised heads: Tn = T D (for Q_k = -V_k T D), Qk = D T D (Q_1 = I - D T D)
    for (int i = tid; i < kDirectB * kDirectB; i += blockDim.x) {
      const int r = i & 31, c = i >> 5;
      const bool in = r < b && c < b;
      const double t = in ? Tn[c * kLd + r] * s_h[c] : 0.0;
      Tn[c * kLd + r] = t;
      Qk[c * kLd + r] = in ? s_h[r] * t : 0.0;
    }
    __syncthreads();
  }
  if (idx == 0) {
    // on leaf 0's path: U_lvl = U_(lvl-1) Q1 with Q1 = I - D T D and U_0 = I
    // (upper triangular), as soon as the child on the path has its product (it
    // then sets its progress to b + 1).  The top node hands its Q1 alone to the
    // root's solver, which has multiplied what lies below it by then.
    double* Ul = a.Pc + (size_t)lvl * b * b;
    const double* Uprev = Ul - (size_t)b * b;
    const bool mul = lvl > 1 && lvl < a.depth;
    if (mul) {
      if (tid == 0) s_okv[0] = h6_wait(a, a.prog + child0, (unsigned)b + 1u);
      __syncthreads();
      if (!s_okv[0]) return;
    }
    if (mul && nch > 1) {
      h4_load(Pb, Uprev, b);
      mm32(Pb, 1, kLd, kSUpper, Qk, 1, kLd, kSUpper, Po, kLd, b, -1.0, Pb);
    }
    for (int i = tid; i < b * b; i += blockDim.x) {
      const int r = i % b, c = i / b;
      double u = r == c ? 1.0 : 0.0;
      if (nch > 1) u = mul ? Po[c * kLd + r] : u - Qk[c * kLd + r];
      else if (mul) u = __ldcg(Uprev + i);
      Ul[i] = u;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) st_release(a.prog + f, (unsigned)b + 1u);
  }
  if (nch > 1) {
    // Q blocks of the node (for forming Y): Q_1 = I - D T D;  Q_k = -V_k T D
    double* Qp = a.Qn + (size_t)f * kFan * b * b;
    for (int i = tid; i < b * b; i += blockDim.x) {
      const int r = i % b, c = i / b;
      Qp[i] = ((r == c) ? 1.0 : 0.0) - ((r <= c) ? Qk[c * kLd + r] : 0.0);
    }
    mm32(S + 32, 1, ld, kSUpper, Tn, 1, kLd, kSUpper, Qp + b * b, b, b, -1.0, nullptr, nch - 1, 32, b * b);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) st_release(a.done + f, 1u);
}

// The root's solver (one extra CTA): leaf 0's block times the product up its
// path below the top node while that node works; once it has published its R
// and its own Q block, the sign-choice LU, T, W and U^-1.
__device__ void h6_root_solver(const Hr4Args& a, double* sm) {
  __shared__ int s_ok;
  const int b = a.b, top = a.base[a.depth];
  double* sX = sm + 3 * kBlk;
  double* sM = sX + kBlk;
  double* sQ = sM + kBlk;
  auto wait = [&](int f) -> bool {
    __syncthreads();
    if (threadIdx.x == 0) s_ok = h6_wait(a, a.prog + f, (unsigned)b + 1u);
    __syncthreads();
    return s_ok != 0;
  };
  if (!wait(0)) return;
  if (a.depth > 1) {
    if (!wait(a.base[a.depth - 1])) return;
    h4_load(sM, a.Pc, b);
    h4_load(sQ, a.Pc + (size_t)(a.depth - 1) * b * b, b);
    mm32(sM, 1, kLd, kSDense, sQ, 1, kLd, kSUpper, sX, kLd, up8(b), 1.0, nullptr);
  } else {
    h4_load(sX, a.Pc, b);
  }
  if (!wait(top)) return;
  h4_root(a, sm);
}

constexpr int kYRows = 64;                 // rows of Y one CTA forms
constexpr int kYLd = kYRows + 1;
constexpr int kYDoubles = 2 * kDirectB * kYLd + 4 * kBlk;

// Columns 8 CB .. 8 CB + 7 of X U for 32 rows (one per lane), U upper
// triangular (ld kLd), X column-major (ld kYLd): init + sign * X U.
template <int CB>
__device__ __forceinline__ void h6_y_cols(const double* X, const double* U, double sign, double (&acc)[8]) {
  double p[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) p[u] = 0.0;
#pragma unroll 4
  for (int k = 0; k < 8 * CB; ++k) {
    const double x = X[k * kYLd];
#pragma unroll
    for (int u = 0; u < 8; ++u) p[u] = fma(x, U[(8 * CB + u) * kLd + k], p[u]);
  }
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const double x = X[(8 * CB + kk) * kYLd];
#pragma unroll
    for (int u = kk; u < 8; ++u) p[u] = fma(x, U[(8 * CB + u) * kLd + 8 * CB + kk], p[u]);
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) acc[u] = fma(sign, p[u], acc[u]);
}

__device__ __forceinline__ void h6_y_mul(int cb, const double* X, const double* U, double sign, double (&acc)[8]) {
  switch (cb) {
    case 0: h6_y_cols<0>(X, U, sign, acc); break;
    case 1: h6_y_cols<1>(X, U, sign, acc); break;
    case 2: h6_y_cols<2>(X, U, sign, acc); break;
    default: h6_y_cols<3>(X, U, sign, acc); break;
  }
}

// Y of 64 rows of a leaf, while the tree still runs.  Launched as the tree
// kernel's programmatic dependent: its CTAs start when every CTA of the tree
// has started, so everything they wait for is running.
//  * the leaf's rows of its explicit Q, Ql = [I; 0] - V (T V_top^T), while the
//    tree works;
//  * B = Q^(1) ... Q^(depth), the Q blocks from the leaf's parent up to the
//    root, each multiplied in as its node finishes;
//  * M = B U^-1 when the root's U^-1 is there, and Y = Ql M: 350 FP64
//    instructions per sub-partition behind the solver for 64 rows, where
//    k_hr4_form_y multiplies the whole path and forms Y after it (38 us and a
//    launch at 8192 x 32).
__device__ void h6_y(const Hr4Args& a, int y, double* sm) {
  __shared__ int s_ok;
  const int b = a.b, tid = threadIdx.x, lane = tid & 31, warp = warp_id();
  const int leaf = y / a.yparts, part = y % a.yparts;
  const size_t nb2 = (size_t)b * b;
  const int64_t r0 = t4_leaf_row0(a.m, a.P, leaf);
  const int L = (int)(t4_leaf_row0(a.m, a.P, leaf + 1) - r0);
  const int p0 = part * kYRows;
  const int n = L - p0 < kYRows ? L - p0 : kYRows;   // rows of this part (none in a short leaf's last part)
  if (n <= 0) return;
  double* sV = sm;
  double* sQ1 = sV + kDirectB * kYLd;
  double* VT = sQ1 + kDirectB * kYLd;
  double* S1 = VT + kBlk;
  double* S2 = S1 + kBlk;
  double* S3 = S2 + kBlk;
  auto wait = [&](int f) -> bool {
    __syncthreads();
    if (tid == 0) s_ok = h6_wait(a, a.done + f, 1u);
    __syncthreads();
    return s_ok != 0;
  };
  if (!wait(leaf)) return;
  for (int e = tid; e < kYRows * kDirectB; e += blockDim.x) {
    const int c = e / kYRows, r = e % kYRows, rl = p0 + r;
    double v = 0.0;
    if (r < n && c < b) v = rl == c ? 1.0 : __ldcg(a.Vw + (int64_t)c * a.m + r0 + rl);
    sV[c * kYLd + r] = v;
  }
  for (int e = tid; e < kDirectB * kDirectB; e += blockDim.x) {
    const int r = e & 31, c = e >> 5;
    double v = 0.0;
    if (r < b && c < b) v = r > c ? __ldcg(a.Vw + (int64_t)c * a.m + r0 + r) : (r == c ? 1.0 : 0.0);
    S1[c * kLd + r] = v;
  }
  h4_load(S2, a.Tl + (size_t)leaf * nb2, b);
  mm32(S2, 1, kLd, kSUpper, S1, kLd, 1, kSUpper, VT, kLd, up8(b), 1.0, nullptr);   // T V_top^T
  // 32 rows x 8 columns per warp; warps w and w + 4 share a sub-partition and
  // take column blocks w and 3 - w, so that the triangle's work is even
  const int g = warp >> 2, cb = g ? 3 - (warp & 3) : warp & 3;
  const int r = 32 * g + lane, rl = p0 + r;
  if (warp < 8 && 8 * cb < b) {
    double acc[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u] = rl == 8 * cb + u ? 1.0 : 0.0;
    h6_y_mul(cb, sV + r, VT, -1.0, acc);
#pragma unroll
    for (int u = 0; u < 8; ++u) sQ1[(8 * cb + u) * kYLd + r] = acc[u];
  }
  // B in S1
  for (int e = tid; e < kDirectB * kDirectB; e += blockDim.x) {
    const int r2 = e & 31, c = e >> 5;
    S1[c * kLd + r2] = (r2 == c && c < b) ? 1.0 : 0.0;
  }
  bool any = false;
  int child = leaf;
  for (int lvl = 1; lvl <= a.depth; ++lvl) {
    const int nd = child / kFan;
    if (h4_children(a, lvl, nd) > 1) {
      if (!wait(a.base[lvl] + nd)) return;
      h4_load(any ? S3 : S1, a.Qn + ((size_t)(a.base[lvl] + nd) * kFan + (child - nd * kFan)) * nb2, b);
      if (any) {
        mm32(S1, 1, kLd, kSUpper, S3, 1, kLd, kSUpper, S2, kLd, up8(b), 1.0, nullptr);
        double* t = S1;
        S1 = S2;
        S2 = t;
      }
      any = true;
    }
    child = nd;
  }
  if (!wait(a.base[a.depth] + 1)) return;   // U^-1
  h4_load(S3, a.Uinv, b);
  mm32(S1, 1, kLd, kSUpper, S3, 1, kLd, kSUpper, S2, kLd, up8(b), 1.0, nullptr);   // M
  if (warp < 8 && 8 * cb < b) {
    double acc[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u] = 0.0;
    h6_y_mul(cb, sQ1 + r, S2, 1.0, acc);
    if (r < n && r0 + rl >= b) {   // the panel's top b rows come from the root
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (8 * cb + u < b) a.A[(int64_t)(8 * cb + u) * a.lda + r0 + rl] = acc[u];
    }
  }
}

__global__ void __launch_bounds__(kLeafThreads, 2) k_hr6_pipe(Hr4Args a) {
  extern __shared__ double sm6[];
  __shared__ double s_h[kDirectB], s_gam[kDirectB];
  __shared__ int s_role;
  if (threadIdx.x == 0) s_role = (int)atomicAdd(a.ticket, 1u);
  __syncthreads();
  // The Y kernel (k_hr6_y) may start once every CTA of this grid has started
  // and the leaves are done: their SMs are then free, one for each of its CTAs
  // (started with the tree, its CTAs shared SMs and took 20 us for 10).
  if (s_role >= a.P) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // flat tree id: leaves 0 .. P-1, the nodes level by level, the root's solver
  const int f = s_role, top = a.base[a.depth];
  if (f < a.P)
    h6_leaf(a, f, sm6, s_h, s_gam);
  else if (f <= top)
    h6_node(a, f, sm6, s_h, s_gam);
  else
    h6_root_solver(a, sm6);
}

__global__ void __launch_bounds__(kLeafThreads, 2) k_hr6_y(Hr4Args a) {
  extern __shared__ double sm6[];
  h6_y(a, (int)blockIdx.x, sm6);
  // this grid ends after the tree's: what follows it in the stream follows both
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The product of the Q blocks along the root-to-node path times U^-1, for
// every node of level lvl (1 <= lvl < depth), from the parents' products:
// M(node) = Q(parent, child index) M(parent), or M(parent) for an only child,
// with M(root) = U^-1.  Run level by level from the top, this forms every
// path product once (about P / 3 products) instead of once per leaf and
// level (P x depth) in k_hr4_form_y.
__global__ void __launch_bounds__(kLeafThreads) k_hr4_node_m(Hr4Args a, int lvl) {
  extern __shared__ double sm4[];
  const int b = a.b, tid = threadIdx.x;
  const int c = blockIdx.x;                 // node index within level lvl
  const int nd = c / kFan;                  // parent at level lvl + 1
  const size_t nb2 = (size_t)b * b;
  const double* Mp = (lvl + 1 == a.depth) ? a.Uinv : a.Mn + (size_t)(a.base[lvl + 1] + nd) * nb2;
  double* Mo = a.Mn + (size_t)(a.base[lvl] + c) * nb2;
  double* sQ = sm4;
  double* sM = sQ + kBlk;
  if (h4_children(a, lvl + 1, nd) > 1) {
    h4_load(sQ, a.Qn + ((size_t)(a.base[lvl + 1] + nd) * kFan + (c - nd * kFan)) * nb2, b);
    h4_load(sM, Mp, b);
    mm32(sQ, 1, kLd, kSUpper, sM, 1, kLd, kSUpper, Mo, b, b, 1.0, nullptr);
  } else {
    for (int idx = tid; idx < b * b; idx += blockDim.x) Mo[idx] = __ldcg(Mp + idx);
  }
}

__global__ void __launch_bounds__(kThreads) k_hr4_form_y(Hr4Args a) {
  extern __shared__ double sm4[];
  const int b = a.b, tid = threadIdx.x;
  const int leaf = blockIdx.x;
  const int64_t r0 = t4_leaf_row0(a.m, a.P, leaf);
  const int64_t r1 = t4_leaf_row0(a.m, a.P, leaf + 1);
  double* sM = sm4;
  double* sX = sM + kBlk;
  double* sY = sX + kBlk;
  double* sT = sY + kBlk;
  // the levels above 1 come from k_hr4_node_m when it ran (a.Mn)
  const int top = (a.Mn && a.depth >= 2) ? 1 : a.depth;
  if (top < a.depth)
    h4_load(sM, a.Mn + (size_t)(a.base[1] + leaf / kFan) * b * b, b);
  else
    h4_load(sM, a.Uinv, b);
  for (int lvl = top; lvl >= 1; --lvl) {
    int nd = leaf;
    for (int l = 0; l < lvl; ++l) nd /= kFan;
    int child = leaf;
    for (int l = 0; l < lvl - 1; ++l) child /= kFan;
    if (h4_children(a, lvl, nd) > 1) {
      const int k = child - nd * kFan;
      h4_load(sX, a.Qn + ((size_t)(a.base[lvl] + nd) * kFan + k) * b * b, b);
      mm32(sX, 1, kLd, kSUpper, sM, 1, kLd, kSUpper, sY, kLd, up8(b), 1.0, nullptr);
      double* t = sM;
      sM = sY;
      sY = t;
    }
  }
  // Z = T (V_top^T M);  Y = [M; 0] - V Z
  for (int idx = tid; idx < kDirectB * kDirectB; idx += blockDim.x) {
    const int r = idx & 31, c = idx >> 5;
    sY[c * kLd + r] = (r < b && c < b) ? (r > c ? a.Vw[(int64_t)c * a.m + r0 + r] : (r == c ? 1.0 : 0.0)) : 0.0;
  }
  h4_load(sT, a.Tl + (size_t)leaf * b * b, b);
  mm32(sY, kLd, 1, kSUpper, sM, 1, kLd, kSUpper, sX, kLd, up8(b), 1.0, nullptr);    // sX = V_top^T M
  mm32(sT, 1, kLd, kSUpper, sX, 1, kLd, kSUpper, sY, kLd, up8(b), 1.0, nullptr);   // sY = Z = T sX
  // Z is upper triangular: Y[r][c] = M[r][c] - sum_{k<=c} V[r][k] Z[k][c], eight
  // columns at a time with independent accumulators (the loops unroll fully,
  // so the triangle is cut at compile time)
  for (int64_t r = r0 + tid; r < r1; r += blockDim.x) {
    if (r < b) continue;
    const int rl = (int)(r - r0);
    double v[kDirectB];
#pragma unroll
    for (int k = 0; k < kDirectB; ++k)
      v[k] = (k < b) ? (rl > k ? a.Vw[(int64_t)k * a.m + r] : (rl == k ? 1.0 : 0.0)) : 0.0;
#pragma unroll
    for (int cb = 0; cb < kDirectB; cb += 8) {
      if (cb < b) {
        double acc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[u] = (rl < b && cb + u < b) ? sM[(cb + u) * kLd + rl] : 0.0;
#pragma unroll
        for (int k = 0; k < cb + 8; ++k) {
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (k <= cb + u) {
              const double z = (cb + u < b) ? sY[(cb + u) * kLd + k] : 0.0;
              acc[u] = fma(-v[k], z, acc[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (cb + u < b) a.A[(int64_t)(cb + u) * a.lda + r] = acc[u];
      }
    }
  }
}

int hr_direct4(double* A, int64_t lda, int64_t m, int b, double* T, int64_t ldT, double* W,
               int64_t ldW, int* d_status, cudaStream_t s) {
  if (b < 1 || b > kDirectB || m < b) return CANDMC_ERR_ARG;
  int64_t want = t_leaf_rows > 0 ? t_leaf_rows : g_leaf_rows > 0 ? g_leaf_rows : kLeafRows;
  // tall panels (throughput, not the latency of one leaf, sets the time) take
  // 256-row leaves unless the knob asks for a height
  if ((t_leaf_rows > 0 || g_leaf_rows == 0) && m >= kTallPanelRows) want = std::max<int64_t>(want, 256);
  // short panels take 64-row leaves while leaves, nodes and the CTAs of Y have
  // an SM each (2048 x 32: 178 us against 196, 512 x 32: 165 against 187)
  const int64_t p64 = (m + 63) / 64;
  if ((t_leaf_rows > 0 ? g_pipe_leaf_rows == 0 : g_leaf_rows == 0) && 2 * p64 + p64 / 3 + 4 <= device_sms()) want = 64;
  const int64_t leaf_rows = std::max<int64_t>(32, std::min<int64_t>(want, 256));
  // leaves of at most leaf_rows rows and at least b rows
  int64_t P = std::max<int64_t>(1, std::min<int64_t>((m + leaf_rows - 1) / leaf_rows, m / b));
  if (P > (1 << 24)) return CANDMC_ERR_ARG;
  Hr4Args a{};
  a.P = (int)P;
  a.nlev[0] = (int)P;
  a.base[0] = 0;
  int total = (int)P, l = 0;
  while (a.nlev[l] > 1) {
    a.nlev[l + 1] = (a.nlev[l] + kFan - 1) / kFan;
    a.base[l + 1] = total;
    total += a.nlev[l + 1];
    ++l;
  }
  a.depth = l;
  const int nnodes = total;
  const int64_t Lmax = (m + P - 1) / P;
  const size_t nb2 = (size_t)b * b;
  // shared block of the leaves:
  // rows padded to the row slots of the factor instantiation that runs (1..4
  // slots of 32 rows, or 8 for leaves of more than 128 rows), and, where the
  // leaf's CTA also works the nodes, at least the 4 x 32 rows of a node
  const int64_t slots = (Lmax + 31) / 32;
  // the pipelined tree while the whole tree is a modest number of CTAs (a
  // latency-bound panel); the level-by-level tree for many leaves, where the
  // leaves dominate and the pipeline would only add synchronisation
  const bool pipe = g_pipe_tree && nnodes <= 4096;
  a.ldS = (int)std::max<int64_t>(32 * (slots <= 4 ? slots : kMaxR), pipe ? 0 : kFan * 32) + 1;
  if (a.ldS > 32 * kMaxR + 1) return CANDMC_ERR_ARG;
  // Y beside the tree (k_hr6_y) while its CTAs find free SMs; with more of
  // them than SMs the FP64 pipes bound the panel, and that form spends 1.8
  // times the instructions of k_hr4_form_y
  const int64_t yparts = (Lmax + kYRows - 1) / kYRows;
  a.yparts = (pipe && P * yparts <= device_sms()) ? (int)yparts : 0;
  const size_t sm = sizeof(double) * std::max<size_t>({(size_t)a.ldS * kDirectB + 2 * kBlk + kLeafScratch,
                                                       (size_t)kNodeDoubles, (size_t)kRootDoubles});
  if (sm > 200 * 1024) return CANDMC_ERR_ARG;
  // one workspace, carved in 256-byte aligned pieces; the counters and the
  // node R blocks (read before all their entries are written) lead it, so
  // one memset clears both
  // counters: cnt (last arriver) or prog + done + ticket + fail (pipelined)
  const size_t ncnt = pipe ? 2 * (size_t)nnodes + 3 : (size_t)nnodes;
  auto rup256 = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t o_cnt = 0;
  const size_t o_rn = o_cnt + rup256(sizeof(unsigned) * ncnt);
  const size_t o_vw = o_rn + rup256(sizeof(double) * nb2 * nnodes);
  const size_t o_tl = o_vw + rup256(sizeof(double) * (size_t)m * b);
  const size_t o_qn = o_tl + rup256(sizeof(double) * nb2 * P);
  const size_t o_uinv = o_qn + rup256(sizeof(double) * nb2 * kFan * nnodes);
  const size_t o_pc = o_uinv + rup256(sizeof(double) * nb2);
  // many leaves: the path products are formed once per node, top down
  const bool node_m = P >= kNodeMinLeaves && a.depth >= 2;
  const size_t o_mn = o_pc + (pipe ? rup256(sizeof(double) * nb2 * (a.depth + 1)) : 0);
  const size_t total_bytes = o_mn + (node_m ? rup256(sizeof(double) * nb2 * nnodes) : 0);
  DevBuf ws;
  CANDMC_RET(ws.alloc(total_bytes, s));
  char* base = static_cast<char*>(ws.p);
  CANDMC_CK(cudaMemsetAsync(base, 0, pipe ? o_vw : o_rn, s));
  a.A = A; a.lda = lda; a.m = m; a.b = b;
  a.Vw = reinterpret_cast<double*>(base + o_vw);
  a.Tl = reinterpret_cast<double*>(base + o_tl);
  a.Rn = reinterpret_cast<double*>(base + o_rn);
  a.Qn = reinterpret_cast<double*>(base + o_qn);
  a.cnt = reinterpret_cast<unsigned*>(base + o_cnt);
  if (pipe) {
    a.prog = a.cnt;
    a.done = a.cnt + nnodes;
    a.ticket = a.cnt + 2 * nnodes + 1;
    a.fail = reinterpret_cast<int*>(a.cnt + 2 * nnodes + 2);
    a.Pc = reinterpret_cast<double*>(base + o_pc);
  }
  a.T = T; a.ldT = ldT; a.W = W; a.ldW = ldW;
  a.Uinv = reinterpret_cast<double*>(base + o_uinv);
  a.Mn = node_m ? reinterpret_cast<double*>(base + o_mn) : nullptr;
  a.status = d_status;
  a.polls = g_panel_polls;
  a.smem_polls = g_panel_smem_polls;
  static std::atomic<bool> attr{false};
  if (!attr) {
    CANDMC_CK(cudaFuncSetAttribute(k_hr4_leaf_tree, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   200 * 1024));
    CANDMC_CK(cudaFuncSetAttribute(k_hr6_pipe, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    CANDMC_CK(cudaFuncSetAttribute(k_hr6_y, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr = true;
  }
  {
    ProfScope ps(CANDMC_KCLASS_PANEL_LEAF, 2.0 * m * b * b, s);
    if (pipe)
      k_hr6_pipe<<<(unsigned)nnodes + 1u, kLeafThreads, sm, s>>>(a);
    else
      k_hr4_leaf_tree<<<(unsigned)P, kLeafThreads, sm, s>>>(a);
  }
  CANDMC_CK(cudaGetLastError());
  if (node_m) {
    for (int lvl = a.depth - 1; lvl >= 1; --lvl) {
      ProfScope ps(CANDMC_KCLASS_PANEL_Y, 2.0 * a.nlev[lvl] * (double)nb2 * b / 3.0, s);
      k_hr4_node_m<<<(unsigned)a.nlev[lvl], kLeafThreads, sizeof(double) * 2 * kBlk, s>>>(a, lvl);
      CANDMC_CK(cudaGetLastError());
    }
  }
  if (a.yparts) {
    ProfScope ps(CANDMC_KCLASS_PANEL_Y, 2.0 * m * b * b, s);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(P * a.yparts));
    cfg.blockDim = dim3(kLeafThreads);
    cfg.dynamicSmemBytes = sizeof(double) * kYDoubles;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CANDMC_CK(cudaLaunchKernelEx(&cfg, k_hr6_y, a));
  } else {
    // with several waves of leaves, one thread per leaf row: leaves of at most
    // 128 rows take 128-thread CTAs, so two of them (252 registers a thread)
    // share an SM; a single wave keeps 256 threads for the path products
    const unsigned ythreads = (Lmax <= 128 && P >= kNodeMinLeaves) ? 128u : (unsigned)kThreads;
    ProfScope ps(CANDMC_KCLASS_PANEL_Y, 2.0 * m * b * b, s);
    k_hr4_form_y<<<(unsigned)P, ythreads, sizeof(double) * 4 * kBlk, s>>>(a);
  }
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

}  // namespace candmc
