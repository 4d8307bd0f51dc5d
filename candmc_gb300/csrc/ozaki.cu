// Emulated-FP64 contractions of the CAQR trailing update on the 5th-generation
// tensor cores (tcgen05, BF16 inputs, FP32 accumulation in TMEM).
//
// Ozaki-style splitting (Ozaki, Ogita, Oishi, Rump, "Error-free transformations
// of matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59, 2012): every operand element x of a
// scale group with |x| < 2^e is written as x = 2^(e-8) * sum_{i<7} d_i 2^(-8i)
// with balanced integer digits |d_0| <= 256, |d_i| <= 128 (i >= 1).  Slice i
// holds d_i * 2^(-8i), exact in BF16 (<= 8 significant bits).  A product of
// two slices has <= 16 significant bits, so a K = 128 sum of one "level"
// L = i + j is an exact FP32 integer (at its weight); levels 0..3 get one TMEM
// accumulator each and levels 4..6 share a fifth (their rounding sits below
// 2^-56 of the result).  28 slice pairs (i + j <= 6) are issued per K step.
//
// The trailing matrix is held as float pairs (hi, lo) ("df64", ~48 bits)
// during the emulated factorization, so no epilogue needs the GB300's slow
// FP64 pipe: the five accumulators are combined exactly (integer/fraction
// split, fast TwoSum), scaled by a power of two and accumulated or subtracted
// in df64.  Finished rows (the panel's R block) are written back as FP64.
//
// Kernel layout: persistent CTAs (at most one per SM) over work items of one
// 128 x 96 output tile and K range each; 14 warps.  k_oz_mma takes operand
// slices from global memory in the UMMA "K-major, no swizzle" core-matrix
// order, so each K16 step of a tile is a contiguous 4 KB (A, 128 rows) and 3 KB
// (B, 96 rows) block per slice: a producer warp streams them with bulk
// asynchronous copies into a 4-stage shared-memory ring, an MMA warp issues the
// 28 tcgen05.mma of a step and commits them to the stage's "empty" mbarrier
// (and, at the end of an exact-accumulation group, to the epilogue's "full"
// mbarrier), and twelve epilogue warps drain and combine the accumulators and
// release them; the read-modify-write of C then overlaps the next group's MMAs.
// k_oz_tn (Y^T C for float pairs) has only A sliced beforehand: its twelve warps
// slice C on the way.  Every wait is bounded; a wait that runs out sets the
// status word, the roles stop, the MMA warp waits for its last MMAs, and the CTA
// frees its TMEM and returns.  Both kernels are kept short: what runs once per
// group costs some 30 cycles an instruction where the loop does not fit the
// instruction cache.
#include <cuda_bf16.h>
#include <math.h>

#include <algorithm>
#include <initializer_list>

#include "kernels.cuh"

namespace candmc {

constexpr int OZ_S = 7;           // slices per operand of the emulated-FP64 form
constexpr int OZ_S32 = 3;         // slices per operand of the FP32 form
constexpr int OZ_M = 128;         // tile rows (TMEM lanes)
constexpr int OZ_N = 96;          // tile columns
constexpr int OZ_STAGES = 4;
constexpr int OZ_ABYTES = OZ_M * 16 * 2;               // one slice, one K16 step
constexpr int OZ_BBYTES = OZ_N * 16 * 2;
// Per slice count S: TMEM accumulator groups G (levels 0..3 exact each, the
// rest shared, for S = 7; one per level for S <= 5), bytes of one ring stage
// and the dynamic shared memory of the kernel.
template <int S>
struct OzCfg {
  static constexpr int G = S >= 5 ? 5 : S;
  static constexpr int STAGE_BYTES = S * (OZ_ABYTES + OZ_BBYTES);
  static constexpr int SMEM = OZ_STAGES * STAGE_BYTES + 1024;
};
constexpr int OZ_WAIT_LIMIT = 1 << 22;                // bounded mbarrier polls
int g_oz_polls = OZ_WAIT_LIMIT;                       // those of the roles on one another (knob "oz_polls")

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ------------------------------------------------------------------ df64
struct f2 {
  float h, l;
};

__device__ __forceinline__ f2 two_sum(float a, float b) {
  float s = a + b;
  float bb = s - a;
  float e = (a - (s - bb)) + (b - bb);
  return {s, e};
}

__device__ __forceinline__ f2 fast_two_sum(float a, float b) {
  float s = a + b;
  return {s, b - (s - a)};
}

// x + y
__device__ __forceinline__ f2 df_add(f2 x, f2 y) {
  f2 s = two_sum(x.h, y.h);
  f2 t = two_sum(x.l, y.l);
  s.l += t.h;
  s = fast_two_sum(s.h, s.l);
  s.l += t.l;
  return fast_two_sum(s.h, s.l);
}

// x as FP32 hi + lo, each rounded to nearest even.  A conversion or an addition
// of doubles costs a slot of the FP64 pipe (65 cycles a warp on each
// sub-partition: four of them per element held the conversion at 2.2 TB/s), so in
// the range where both parts are normal the split works on the bits: hi is the
// significand rounded to 24 bits, lo the exact difference of the two bit
// patterns (an integer below 2^28 in units of 2^(e - 52)).
__device__ __forceinline__ f2 df_from_double(double x) {
  const unsigned hw = (unsigned)__double2hiint(x);
  const unsigned long long u = ((unsigned long long)(hw & 0x7fffffffu) << 32) | (unsigned)__double2loint(x);
  const int E = (int)(hw >> 20) & 0x7ff;
  if (E >= 1023 - 70 && E < 1023 + 127) {
    const unsigned long long t = (u + 0x0fffffffull + ((u >> 29) & 1ull)) >> 29;
    const int d = (int)(unsigned)(u - (t << 29));
    const unsigned sign = hw & 0x80000000u;
    const float h = __uint_as_float(((unsigned)t - (896u << 23)) | sign);
    const float l = __fmul_rn((float)d, __uint_as_float(((unsigned)(E - 1023 - 52 + 127) << 23) | sign));
    return {h, l};
  }
  if (u == 0) return {__uint_as_float(hw), 0.0f};
  float h = (float)x;
  float l = (float)(x - (double)h);
  return {h, l};
}

// A float as a double by its bits (no FP64 conversion): a subnormal is scaled to
// a normal float first, and the exponent of an infinity or NaN becomes the double's.
__device__ __forceinline__ double widen(float f) {
  const bool sub = (__float_as_uint(f) & 0x7f800000u) == 0;
  const unsigned i = __float_as_uint(sub ? __fmul_rn(f, 18446744073709551616.0f) : f), m = i & 0x7fffffffu;   // 2^64
  unsigned h = (m >> 3) + (sub ? 0x38000000u - (64u << 20) : 0x38000000u);
  if (m >= 0x7f800000u) h += 0x38000000u;
  if (m == 0) h = 0;
  return __hiloint2double((int)(h | (i & 0x80000000u)), (int)(i << 29));
}

__device__ __forceinline__ double df_to_double(f2 x) { return widen(x.h) + widen(x.l); }

// Two floats in one 64-bit register: the f32x2 instructions round each half
// as the scalar ones do and take one issue slot for both.
struct f2x2 {
  unsigned long long v;
};
__device__ __forceinline__ f2x2 pack2(float a, float b) {
  f2x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f2x2 x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x.v));
  return r;
}
__device__ __forceinline__ f2x2 add2(f2x2 a, f2x2 b) {
  f2x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2x2 mul2(f2x2 a, f2x2 b) {
  f2x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2x2 sub2(f2x2 a, f2x2 b) {   // a - b, rounded once
  f2x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(b.v), "l"(0xbf800000bf800000ull), "l"(a.v));
  return r;
}

// ------------------------------------------------------------------ slicing
// 2^e for -126 <= e <= 127 (a normal float): x * pow2f(e) rounds once, as
// ldexpf(x, e) does
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }

// Scale exponent of a group maximum: smallest e with max < 2^e (0 for 0 and for
// an infinity), from the bits (frexpf took 700 cycles where it stands between
// two groups of a contraction).
__device__ __forceinline__ int scale_exp(float mx) {
  const unsigned b = __float_as_uint(mx);
  if (!(mx > 0.0f) || b >= 0x7f800000u) return 0;
  return b >= 0x00800000u ? (int)(b >> 23) - 126 : 32 - __clz((int)b) - 149;
}

// The S digits of two values (p + q scaled below 2^8, |q| at most half an ulp
// of p), each at its natural weight 2^(-8i): digit i is the rest rounded to a
// multiple of that weight by adding and taking away 1.5 * 2^(23 - 8i), and the
// rest stays exact.  The low word comes in before every second digit: a rest
// below 2^(-8i-1) and a q below half an ulp of it are still balanced digits.
// put(i, d) takes the digits of both values.
template <int S, class Put>
__device__ __forceinline__ void slice_digits(f2x2 p, f2x2 q, Put put) {
#pragma unroll
  for (int i = 0; i < S; ++i) {
    if (i > 0 && i == S - 1) {
      p = add2(p, q);
    } else if (i > 0 && i % 2 == 0) {
      const f2x2 t = add2(p, q);
      q = sub2(q, sub2(t, p));
      p = t;
    }
    const float m = 12582912.0f * __int_as_float((127 - 8 * i) << 23);
    const f2x2 shift = pack2(m, m);
    const f2x2 d = sub2(add2(p, shift), shift);
    put(i, d);
    if (i + 1 < S) p = sub2(p, d);
  }
}

// Two digits as BF16: they have at most 8 significant bits, so the upper halves
// of the floats are exact (a conversion takes a quarter-rate slot, this a byte
// permutation; a NaN keeps its quiet bit there).
__device__ __forceinline__ uint32_t to_bf16x2(f2x2 v) {
  const float2 w = unpack2(v);
  return __byte_perm(__float_as_uint(w.x), __float_as_uint(w.y), 0x7632);
}

struct SliceSrc {
  const double* d;     // FP64 source (mask applies), or nullptr
  const float2* df;    // df64 source, or nullptr
  int64_t ld;
  int mask;            // kDense / kUnitLower / kUpper (FP64 source)
  int64_t off;         // diagonal offset of the mask
};

__device__ __forceinline__ f2 src_at(const SliceSrc& s, int64_t r, int64_t c) {
  if (s.df) {
    float2 v = s.df[c * s.ld + r];
    return {v.x, v.y};
  }
  double x;
  switch (s.mask) {
    case kUnitLower: x = (r > c + s.off) ? s.d[c * s.ld + r] : (r == c + s.off ? 1.0 : 0.0); break;
    case kUpper: x = (r <= c + s.off) ? s.d[c * s.ld + r] : 0.0; break;
    case kLower: x = (r >= c + s.off) ? s.d[c * s.ld + r] : 0.0; break;
    default: x = s.d[c * s.ld + r];
  }
  return df_from_double(x);
}

// Slices of an R x K operand (rows n, the contraction index k), with one scale
// exponent per row and K group of G (a multiple of 16, at most 128).  Element
// (n, k) is src(k, n) (krow = 0: K runs down the source's columns) or
// src(n, k) (krow = 1: K runs along its rows); rows from Nvalid to Rpad
// and k from Kvalid on are zero.  Slices: S planes of Rpad x Kpad in the
// core-matrix order; exponents e[(k / G) * Rpad + n].  A launch takes up to three
// operands, one block range each: those of a panel's own products are small,
// and the second and third launch cost 9 us each beside a first of 10.
// A CTA takes kSliceRows rows and one group: it stages the group in shared
// memory, warp w finds the exponents of rows 2w and 2w + 1, and then the
// 16 x 16 elements of K16 block w are, in every plane, one contiguous 512-byte
// run, of which a lane writes the 16 bytes of 8 consecutive k.  The rows' pitch
// shifts a row by 16 bytes, so the lanes' 16-byte reads (8 rows at one k)
// fall on different banks.  Bound by memory (8 bytes read and 2 S written per
// element) once the digits take some 15 issue slots: at about 100, one TwoSum
// for each, 16384 x 8192 elements took 599 us, with 8-way bank conflicts.
constexpr int kSliceRows = 16;

struct SliceJob {
  SliceSrc src;
  int krow;
  int64_t Kvalid, Nvalid, Rpad, Kpad;
  int G;
  __nv_bfloat16* out;
  int* e;
  unsigned blocks() const { return (unsigned)((Rpad + kSliceRows - 1) / kSliceRows * (Kpad / G)); }
};
struct SliceJobs {
  SliceJob job[3];
  unsigned end[3];   // first block after each job's
};

template <int S>
__global__ void __launch_bounds__(256) k_slice(const __grid_constant__ SliceJobs jobs) {
  __shared__ __align__(16) float2 tile[kSliceRows][128 + 2];
  __shared__ int s_e[kSliceRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int jb = blockIdx.x < jobs.end[0] ? 0 : blockIdx.x < jobs.end[1] ? 1 : 2;
  const SliceJob& J = jobs.job[jb];
  const unsigned block = blockIdx.x - (jb ? jobs.end[jb - 1] : 0);
  const SliceSrc& src = J.src;
  const int64_t Kvalid = J.Kvalid, Nvalid = J.Nvalid, Rpad = J.Rpad, Kpad = J.Kpad;
  const int G = J.G;
  const unsigned nblocks = (unsigned)((Rpad + kSliceRows - 1) / kSliceRows);
  const int64_t n0 = (int64_t)(block % nblocks) * kSliceRows;
  const int64_t g = block / nblocks, kb0 = g * G;
  if (J.krow) {
    const int r = threadIdx.x & 15;
    f2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = (threadIdx.x >> 4) + 16 * u;
      v[u] = {0.0f, 0.0f};
      if (k < G && n0 + r < Nvalid && kb0 + k < Kvalid) v[u] = src_at(src, n0 + r, kb0 + k);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) tile[r][(threadIdx.x >> 4) + 16 * u] = make_float2(v[u].h, v[u].l);
  } else {
    f2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int64_t n = n0 + 2 * warp + (u >> 2);
      const int k = lane + 32 * (u & 3);
      v[u] = {0.0f, 0.0f};
      if (k < G && n < Nvalid && kb0 + k < Kvalid) v[u] = src_at(src, kb0 + k, n);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) tile[2 * warp + (u >> 2)][lane + 32 * (u & 3)] = make_float2(v[u].h, v[u].l);
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = 2 * warp + u;
    float mx = 0.0f;
#pragma unroll
    for (int k = 0; k < 128; k += 32) mx = fmaxf(mx, fabsf(tile[r][k + lane].x));
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    // the lo part can push |x| just above |hi|'s bound; leave one ulp of room
    const int e = scale_exp(mx * (1.0f + 1.0e-6f));
    if (lane == 0) {
      s_e[r] = e;
      if (n0 + r < Rpad) J.e[g * Rpad + n0 + r] = e;
    }
  }
  __syncthreads();
  const int r = (lane >> 4) * 8 + (lane & 7), khalf = (lane >> 3) & 1;
  if (n0 + r >= Rpad || warp >= G / 16) return;
  // 2^(8 - e) as two normal factors, the second one 1 unless e < -119
  const int k1 = min(8 - s_e[r], 127);
  const float f1 = pow2f(k1), f2v = pow2f(8 - s_e[r] - k1);
  const f2x2 sc1 = pack2(f1, f1), sc2 = pack2(f2v, f2v);
  const float4* t4 = reinterpret_cast<const float4*>(&tile[r][warp * 16 + khalf * 8]);
  uint32_t d[S][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float4 x = t4[c];
    slice_digits<S>(mul2(mul2(pack2(x.x, x.z), sc1), sc2), mul2(mul2(pack2(x.y, x.w), sc1), sc2),
                    [&](int i, f2x2 v) { d[i][c] = to_bf16x2(v); });
  }
  const int64_t plane = Rpad * Kpad;
  __nv_bfloat16* o = J.out + ((kb0 >> 4) + warp) * (Rpad * 16) + ((n0 >> 3) + (lane >> 4)) * 128 + khalf * 64 + (lane & 7) * 8;
#pragma unroll
  for (int i = 0; i < S; ++i)
    *reinterpret_cast<uint4*>(o + i * plane) = make_uint4(d[i][0], d[i][1], d[i][2], d[i][3]);
}

// ------------------------------------------------------------------ tcgen05 kernel
struct OzArgs {
  const __nv_bfloat16* As;   // A-operand slices: S planes of AR x Kpad
  int64_t AR;
  const __nv_bfloat16* Bs;   // k_oz_mma: B-operand slices, S planes of BR x Kpad
  int64_t BR;
  int Kpad;                  // multiple of 16 (k_oz_tn: of 128)
  int k_per_cta;             // K extent of one work item (multiple of kgroup)
  int kgroup;                // K rows per scale group / accumulator readout (k_oz_tn: 128)
  const int* eA;             // [Kpad / kgroup][AR]
  const int* eB;             // k_oz_mma: [Kpad / kgroup][BR]
  float2* part;              // sums: [split][Nvalid][AR] (ld AR per column), df64 sums over an item's K range
  float2* C;                 // float pairs (ld ldc): k_oz_tn's B operand, kOzPairs' C
  double* C64;               // kOzDoubles: C
  int64_t ldc;
  int64_t Mvalid, Nvalid;
  int64_t Kvalid;            // k_oz_tn: rows of C
  int64_t fp64_rows;         // kOzPairs: rows < fp64_rows are written as FP64 (final)
  int c_assign;              // kOzDoubles: C = product (C is not read)
  int* status;
  int polls;                 // limit of the roles' waits on one another
  int n_mt, n_nt, n_ks;      // work items: M tiles x N tiles x K splits
};

__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  // K-major, no swizzle: LBO = 128 B (next 8 K elements), SBO = 256 B (next 8 rows)
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(128 >> 4) << 16) |
         ((uint64_t)(256 >> 4) << 32) | (1ull << 46);
}

// tcgen05.ld writes its registers asynchronously: they hold the TMEM values
// only after tcgen05.wait::ld.  The compiler sees no dependence between the
// two, so the loaded registers are passed through tmem_regs_ready (an empty
// asm ordered after the wait) before any use.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                 "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_regs_ready(uint32_t* r) {
  asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
               "+r"(r[7]));
}


constexpr int OZ_EPI_WARPS = 12;                     // epilogue warps: 4 TMEM lane quarters x column parts
constexpr int OZ_EPI_COLS = OZ_N * 4 / OZ_EPI_WARPS;  // accumulator columns per epilogue warp
constexpr int OZ_WARPS = 2 + OZ_EPI_WARPS;             // producer, MMA issuer, epilogue
constexpr int OZ_THREADS = OZ_WARPS * 32;
static_assert(OZ_EPI_WARPS % 4 == 0 && OZ_EPI_COLS == 32, "epilogue split: one column per lane for the exponents");

// two df64 values: high words, low words
struct df2 {
  f2x2 h, l;
};

// The accumulators of two output elements (columns j, j + 1 of gr) as df64
// values.  Groups 0..3 hold the diagonals i + j = g of the slice products,
// exact multiples of 2^-8g with |g0| <= 2^23, |g1| <= 2^15, |g2| <= 2^8,
// |g3| < 1 (digits of at most 8 bits over a 128-row group); group 4 holds the
// rest, down to about 2^-40.  Rounding g1 and g2 to integers and g3 to a
// multiple of 2^-16 (the 1.5 * 2^23 and 1.5 * 2^7 shifts) splits them exactly:
// H = g0 + [g1] + [g2] is an integer below 2^24, M = frac(g1) + frac(g2) + [g3]
// a multiple of 2^-16 below 2 in magnitude, both exact, and only
// L = (g3 - [g3]) + g4 rounds.  The two fast TwoSums are exact here (H is zero
// or at least 1 in magnitude), so the result carries about 2^-47 relative
// error, as a df64 sum of the five.  The FP32 form (G < 5, one group per level,
// FP32 accuracy wanted) takes their FP32 sum.
template <int G>
__device__ __forceinline__ df2 combine2(const uint32_t (&gr)[G][8], int j) {
  f2x2 g[G];
#pragma unroll
  for (int q = 0; q < G; ++q) g[q] = pack2(__uint_as_float(gr[q][j]), __uint_as_float(gr[q][j + 1]));
  if constexpr (G == 5) {
    const f2x2 shift = pack2(12582912.0f, 12582912.0f);   // 1.5 * 2^23: rounds to an integer
    const f2x2 shift3 = pack2(192.0f, 192.0f);            // 1.5 * 2^7: rounds to a multiple of 2^-16
    const f2x2 r1 = sub2(add2(g[1], shift), shift);
    const f2x2 r2 = sub2(add2(g[2], shift), shift);
    const f2x2 r3 = sub2(add2(g[3], shift3), shift3);
    const f2x2 H = add2(add2(g[0], r1), r2);
    const f2x2 M = add2(add2(sub2(g[1], r1), sub2(g[2], r2)), r3);
    const f2x2 L = add2(sub2(g[3], r3), g[4]);
    const f2x2 s = add2(H, M);
    const f2x2 l = add2(sub2(M, sub2(s, H)), L);
    const f2x2 h = add2(s, l);
    return {h, sub2(l, sub2(h, s))};
  } else {
    f2x2 h = g[G - 1];
#pragma unroll
    for (int q = G - 2; q >= 0; --q) h = add2(g[q], h);
    return {h, {0ull}};
  }
}

// Accumulation of the epilogue, x + y without the lo-part TwoSum: relative
// error of order 2^-46 of |x| + |y|.  For the FP32 form (G < 5, products
// accurate to FP32) plain FP32, which keeps C in the df64 slots with a zero
// low word.
template <int G>
__device__ __forceinline__ df2 oz_accumulate(df2 x, df2 y) {
  const f2x2 s = add2(x.h, y.h);
  if constexpr (G != 5) return {s, {0ull}};
  const f2x2 bb = sub2(s, x.h);
  const f2x2 e = add2(sub2(x.h, sub2(s, bb)), sub2(y.h, bb));
  const f2x2 l = add2(e, add2(x.l, y.l));
  const f2x2 h = add2(s, l);
  return {h, sub2(l, sub2(h, s))};
}

// C - p for the read-modify-write of float pairs, as df_add of C and -p does it
// (same split by form)
template <int G>
__device__ __forceinline__ df2 oz_subtract(df2 c, df2 p) {
  if constexpr (G != 5) return {sub2(add2(c.h, c.l), p.h), {0ull}};
  const f2x2 s = sub2(c.h, p.h), sb = sub2(s, c.h);
  const f2x2 e = sub2(sub2(c.h, sub2(s, sb)), add2(p.h, sb));
  const f2x2 t = sub2(c.l, p.l), tb = sub2(t, c.l);
  const f2x2 te = sub2(sub2(c.l, sub2(t, tb)), add2(p.l, tb));
  const f2x2 e1 = add2(e, t);
  const f2x2 s1 = add2(s, e1);
  const f2x2 e2 = add2(sub2(e1, sub2(s1, s)), te);
  const f2x2 h = add2(s1, e2);
  return {h, sub2(e2, sub2(h, s1))};
}

// v * 2^e for e beyond the normal floats' range (e >= -312 for float inputs):
// three normal factors, so the partial products stay exact unless the result
// leaves the range
__device__ __forceinline__ float scale_wide(float v, int e) {
  const int e1 = min(max(e, -126), 127), e2 = min(max(e - e1, -126), 127);
  return __fmul_rn(__fmul_rn(__fmul_rn(v, pow2f(e1)), pow2f(e2)), pow2f(e - e1 - e2));
}

__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes)
               : "memory");
}

// bulk global -> shared copy (16-byte aligned, multiple of 16 bytes) that
// signals the byte count on the stage's mbarrier
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, unsigned bytes, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(smem_u32(b))
      : "memory");
}

// Bounded wait of a whole warp.  Warp collectives (votes, elections, TMEM loads) follow
// on either outcome, so the lanes vote on it: all of them leave by the same poll with
// the same result.  A role whose partner has given up runs out by itself: a look at
// the flag in the loop is code at every wait, and these kernels are bound by it.
__device__ __forceinline__ bool oz_wait(uint64_t* b, uint32_t parity, volatile int* fail, int polls) {
  const uint32_t addr = smem_u32(b);
#pragma unroll 1
  for (int it = 0; it < polls; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (__all_sync(0xffffffffu, done)) return true;
  }
  *fail = 1;
  __syncwarp();
  return false;
}

// The last of the `fills` fills of each of n stages has arrived (a bounded wait of the
// producer's warp): a CTA that gave up must not end with copies into it in flight.
__device__ __forceinline__ void oz_copies_done(uint64_t* full, int n, int fills) {
  volatile int unused = 0;
  for (int st = 0; st < n && st < fills; ++st)
    oz_wait(&full[st], (uint32_t)((fills - 1 - st) / n & 1), &unused, OZ_WAIT_LIMIT);
}

// Where a product of slice A_i stands among the products of A_i in one step:
// the first one fills the tensor core's A collector, the others reuse it.
enum OzCollect { kOzSingle, kOzFill, kOzUse, kOzLast };

// One 128 x 96 x 16 BF16 MMA into the accumulator at TMEM column address dt;
// accum = 0 overwrites it.  The whole warp calls it, one elected lane issues:
// in a branch on the lane index the operands go through the vector registers
// and an MMA takes 50 cycles to issue at any width, here 24 (N = 32).
template <OzCollect U>
__device__ __forceinline__ void umma_bf16(uint32_t dt, uint64_t ad, uint64_t bd, uint32_t idesc,
                                          uint32_t accum) {
#define OZ_UMMA(COLLECT)                                                                            \
  asm volatile(                                                                                     \
      "{\n\t.reg .pred p, one;\n\telect.sync _|one, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"       \
      "@one tcgen05.mma.cta_group::1.kind::f16" COLLECT " [%0], %1, %2, %3, p;\n\t}" ::"r"(dt),    \
      "l"(ad), "l"(bd), "r"(idesc), "r"(accum)                                                      \
      : "memory")
  if constexpr (U == kOzFill) OZ_UMMA(".collector::a::fill");
  else if constexpr (U == kOzUse) OZ_UMMA(".collector::a::use");
  else if constexpr (U == kOzLast) OZ_UMMA(".collector::a::lastuse");
  else OZ_UMMA("");
#undef OZ_UMMA
}

// arrives on b once every MMA issued so far has completed (one elected lane)
__device__ __forceinline__ void umma_commit(uint64_t* b) {
  asm volatile(
      "{\n\t.reg .pred one;\n\telect.sync _|one, 0xffffffff;\n\t"
      "@one tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(
          smem_u32(b))
      : "memory");
}

// The slice-pair MMAs of one K16 step.  da / db: descriptors of the stage's
// first A and B slice (the slices follow at fixed byte strides, and a
// descriptor's address field is the shared-memory address / 16, so slice
// descriptors are the base plus a constant).  In loop order the first product
// of accumulator group g is (0, g): with accum = 0 (a group's first step)
// those overwrite their accumulator, every other product adds to it.  The
// products of one A slice follow one another and take it from the collector:
// without that a 128 x 96 x 16 MMA is bound by its 7 KB of operand reads (58
// cycles instead of 50; its multiplications take 48).
template <int S, int G, int I = 0, int J = 0>
__device__ __forceinline__ void oz_issue_step(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc,
                                              uint32_t accum) {
  constexpr int g = (I + J < G - 1) ? I + J : G - 1;
  constexpr OzCollect u = (I == S - 1) ? kOzSingle : (J == 0) ? kOzFill : (J == S - 1 - I) ? kOzLast : kOzUse;
  umma_bf16<u>(tmem + (uint32_t)(g * OZ_N), da + (uint64_t)(I * (OZ_ABYTES >> 4)),
               db + (uint64_t)(J * (OZ_BBYTES >> 4)), idesc, (I == 0 && J < G) ? accum : 1u);
  if constexpr (I + J + 1 < S) oz_issue_step<S, G, I, J + 1>(tmem, da, db, idesc, accum);
  else if constexpr (I + 1 < S) oz_issue_step<S, G, I + 1, 0>(tmem, da, db, idesc, accum);
}

__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}

// Work item w of a launch: (M tile, N tile, K range).  M tiles run fastest so
// that consecutive items of a CTA share the B operand's slices in L2.
struct OzItem {
  int64_t m0, n0;
  int kbeg, kend;
  int split;
};

__device__ __forceinline__ OzItem oz_item(const OzArgs& a, int w) {
  OzItem it;
  const unsigned rest = (unsigned)w / (unsigned)a.n_mt, mt = (unsigned)w % (unsigned)a.n_mt;
  const unsigned ks = rest / (unsigned)a.n_nt, nt = rest % (unsigned)a.n_nt;
  it.m0 = (int64_t)mt * OZ_M;
  it.n0 = (int64_t)nt * OZ_N;
  it.kbeg = (int)ks * a.k_per_cta;
  it.kend = min(it.kbeg + a.k_per_cta, a.Kpad);
  it.split = (int)ks;
  return it;
}

// Read one group's accumulators (columns of this warp from TMEM address taddr,
// 8 at a time), scale them by 2^(eA + eB - 16) and set acc to them (ADD =
// false) or add them to it.  ebs: the columns' exponents shifted to where a
// float has its exponent, so that a scale takes one addition; eb: this lane's
// column's exponent, for one warp-uniform test that every scale is a normal
// float.
template <int G, bool ADD>
__device__ __forceinline__ void oz_drain(uint32_t taddr, const int* ebs, int eb, int eA, df2 (&acc)[OZ_EPI_COLS / 2]) {
  const int eb_min = __reduce_min_sync(0xffffffffu, eb), eb_max = __reduce_max_sync(0xffffffffu, eb);
  const bool normal = __all_sync(0xffffffffu, eA + eb_min - 16 >= -126 && eA + eb_max - 16 <= 127);
  const int fA = (eA - 16 + 127) << 23;
  if (!normal) {
    // one column at a time, the sums in local memory: short code for a rare case (the
    // unrolled form of both cases did not fit the instruction cache)
    float2 x[OZ_EPI_COLS];
#pragma unroll
    for (int j = 0; j < OZ_EPI_COLS; j += 2) {
      const float2 h = unpack2(acc[j / 2].h), l = unpack2(acc[j / 2].l);
      x[j] = make_float2(h.x, l.x);
      x[j + 1] = make_float2(h.y, l.y);
    }
#pragma unroll 1
    for (int j = 0; j < OZ_EPI_COLS; ++j) {
      uint32_t gr[G][8];
#pragma unroll
      for (int g = 0; g < G; ++g) tmem_ld8(taddr + (uint32_t)(g * OZ_N + (j & ~7)), gr[g]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int g = 0; g < G; ++g) {
        tmem_regs_ready(gr[g]);
#pragma unroll
        for (int c = 1; c < 8; ++c)
          if (c == (j & 7)) gr[g][0] = gr[g][c];
      }
      const df2 v = combine2<G>(gr, 0);
      const int e = eA + (ebs[j] >> 23) - 16;
      const df2 sv = {pack2(scale_wide(unpack2(v.h).x, e), 0.0f), pack2(scale_wide(unpack2(v.l).x, e), 0.0f)};
      const df2 r = ADD ? oz_accumulate<G>({pack2(x[j].x, 0.0f), pack2(x[j].y, 0.0f)}, sv) : sv;
      x[j] = make_float2(unpack2(r.h).x, unpack2(r.l).x);
    }
#pragma unroll
    for (int j = 0; j < OZ_EPI_COLS; j += 2)
      acc[j / 2] = {pack2(x[j].x, x[j + 1].x), pack2(x[j].y, x[j + 1].y)};
    return;
  }
#pragma unroll
  for (int c8 = 0; c8 < OZ_EPI_COLS / 8; ++c8) {
    uint32_t gr[G][8];
#pragma unroll
    for (int g = 0; g < G; ++g) tmem_ld8(taddr + (uint32_t)(g * OZ_N + c8 * 8), gr[g]);
    int f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = ebs[c8 * 8 + j];
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int g = 0; g < G; ++g) tmem_regs_ready(gr[g]);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      df2 v = combine2<G>(gr, j);
      const f2x2 sc = pack2(__int_as_float(fA + f[j]), __int_as_float(fA + f[j + 1]));
      v = {mul2(v.h, sc), mul2(v.l, sc)};
      df2& x = acc[c8 * 4 + j / 2];
      x = ADD ? oz_accumulate<G>(x, v) : v;
    }
  }
}

// an item's sums: this lane's row, this warp's columns
__device__ __forceinline__ void oz_store_sums(const OzArgs& a, const OzItem& it, int row, int part,
                                              const df2 (&acc)[OZ_EPI_COLS / 2]) {
  const int64_t gn0 = it.n0 + part * OZ_EPI_COLS;
  float2* out = a.part + ((int64_t)it.split * a.Nvalid + gn0) * a.AR + row;
#pragma unroll
  for (int j = 0; j < OZ_EPI_COLS; ++j) {
    const float2 h = unpack2(acc[j / 2].h), l = unpack2(acc[j / 2].l);
    if (row < a.AR && gn0 + j < a.Nvalid) out[j * a.AR] = (j & 1) ? make_float2(h.y, l.y) : make_float2(h.x, l.x);
  }
}

// What k_oz_mma does with the products: sums over an item's K range (the Y^T C
// of a panel's own FP64 columns), C -= product for float pairs, and C -= product
// or C = product for FP64 storage.
enum OzEpilogue { kOzSums, kOzPairs, kOzDoubles };

// Contraction of two pre-sliced operands: persistent, warp-specialised.  Warp 0
// streams their K16 blocks into a ring of OZ_STAGES stages with bulk copies; warp
// 1 issues the 28 slice-pair MMAs of a stage into the five TMEM accumulator groups
// and commits them (freeing the stage, and at the end of an exact-accumulation
// group, handing the accumulators to the epilogue); the epilogue warps 2.. read
// the accumulators (warp w owns TMEM lanes 32 (w % 4) .. +31 and column part
// (w - 2) / 4), release them, and combine them in df64.  Bound by the MMAs (1390
// cycles a K16 step) and the readout between groups (3100, FP32 additions).  One
// kernel per epilogue: with all of them in one it was 165 KB of instructions
// beside a 32 KB cache, and C -= Y Z' at 16384 x 8192 x 128 took 707 us, now 620.
template <int S, OzEpilogue E>
__global__ void __launch_bounds__(OZ_THREADS, 1) k_oz_mma(OzArgs a) {
  constexpr int G = OzCfg<S>::G;
  constexpr int STAGE_BYTES = OzCfg<S>::STAGE_BYTES;
  extern __shared__ __align__(1024) unsigned char oz_smem[];
  __shared__ __align__(8) uint64_t full_b[OZ_STAGES], empty_b[OZ_STAGES], acc_full, acc_empty, fin;
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int s_fail;
  __shared__ int s_eb[OZ_EPI_WARPS][OZ_EPI_COLS];   // per epilogue warp: its columns' exponents
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  unsigned char* ring = (unsigned char*)(((uintptr_t)oz_smem + 1023) & ~(uintptr_t)1023);
  const int nitems = a.n_mt * a.n_nt * a.n_ks;
  const int steps_per_group = a.kgroup / 16;

  if (tid == 0) {
    for (int st = 0; st < OZ_STAGES; ++st) {
      mbar_init(&full_b[st], 1);
      mbar_init(&empty_b[st], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, OZ_EPI_WARPS);
    mbar_init(&fin, 1);
    s_fail = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_s)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // An A operand of fewer than 128 rows (a narrow Y^T, stored with AR rows)
  // fills only the first AR x 32 bytes of each slice block; the rest of every
  // stage's A blocks is zeroed once here and never written again, so the
  // 128-row MMA reads zeros there.
  if (E == kOzSums && a.AR < OZ_M) {
    const int abytes = (int)a.AR * 32;
    const int tail = (OZ_ABYTES - abytes) / 16;
    for (int idx = tid; idx < OZ_STAGES * S * tail; idx += blockDim.x) {
      const int blk = idx / tail, q = idx % tail;
      *reinterpret_cast<uint4*>(ring + (size_t)(blk / S) * STAGE_BYTES + (size_t)(blk % S) * OZ_ABYTES + abytes +
                                16 * q) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;

  if (warp == 0) {
    // ---------------- producer: the whole warp walks the stages, one elected lane copies
    const int abytes = (E == kOzSums && a.AR < OZ_M) ? (int)a.AR * 32 : OZ_ABYTES;
    const int64_t aplane = a.AR * a.Kpad, bplane = a.BR * a.Kpad;
    int st = 0, fills = 0;
    uint32_t parity = 1;
    bool ok = true;
    for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const OzItem it = oz_item(a, w);
      const __nv_bfloat16* as = a.As + (int64_t)it.kbeg * a.AR + it.m0 * 16;
      const __nv_bfloat16* bs = a.Bs + (int64_t)it.kbeg * a.BR + it.n0 * 16;
      for (int k = it.kbeg; k < it.kend; k += 16) {
        ok = oz_wait(&empty_b[st], parity, &s_fail, a.polls);
        if (!ok) break;
        ++fills;
        if (elect_one()) {
          mbar_expect_tx(&full_b[st], (unsigned)(S * (abytes + OZ_BBYTES)));
          const uint32_t sa = smem_u32(ring + (size_t)st * STAGE_BYTES), sb = sa + S * OZ_ABYTES;
#pragma unroll
          for (int sl = 0; sl < S; ++sl) {
            bulk_g2s(sa + sl * OZ_ABYTES, as + sl * aplane, (unsigned)abytes, &full_b[st]);
            bulk_g2s(sb + sl * OZ_BBYTES, bs + sl * bplane, (unsigned)OZ_BBYTES, &full_b[st]);
          }
        }
        __syncwarp();
        as += a.AR * 16;
        bs += a.BR * 16;
        if (++st == OZ_STAGES) {
          st = 0;
          parity ^= 1;
        }
      }
    }
    oz_copies_done(full_b, OZ_STAGES, fills);
  } else if (warp == 1) {
    // ---------------- MMA issuer: the whole warp walks the stages, one elected lane issues
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_N >> 3) << 17) |
                           ((uint32_t)(OZ_M >> 4) << 24);
    // ring stages are 1024-byte aligned and the ring ends below 256 KB, so
    // base + offset / 16 stays inside the descriptor's 14-bit address field
    const uint64_t ring_desc = make_desc(smem_u32(ring));
    static_assert((OZ_STAGES * STAGE_BYTES + 2048) < (1 << 18), "ring within the descriptor's range");
    static_assert(STAGE_BYTES % 16 == 0 && OZ_ABYTES % 16 == 0 && OZ_BBYTES % 16 == 0, "16-byte strides");
    int st = 0;
    uint32_t parity = 0, acc_parity = 1;
    bool ok = true;
    for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const OzItem it = oz_item(a, w);
      for (int left = (it.kend - it.kbeg) >> 4; left > 0 && ok; left -= steps_per_group) {
        const int steps = min(left, steps_per_group);
        // the epilogue has read the previous group's accumulators
        ok = oz_wait(&acc_empty, acc_parity, &s_fail, a.polls);
        acc_parity ^= 1;
        for (int t = 0; t < steps && ok; ++t) {
          ok = oz_wait(&full_b[st], parity, &s_fail, a.polls);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = ring_desc + (uint64_t)(st * (STAGE_BYTES >> 4));
          oz_issue_step<S, G>(tmem, da, da + (uint64_t)((S * OZ_ABYTES) >> 4), idesc, t > 0 ? 1u : 0u);
          umma_commit(&empty_b[st]);   // the stage is free once these MMAs have read it
          if (++st == OZ_STAGES) {
            st = 0;
            parity ^= 1;
          }
        }
        if (ok) umma_commit(&acc_full);
      }
    }
    // every MMA this warp issued has completed before TMEM is released
    umma_commit(&fin);
    volatile int dummy = 0;
    oz_wait(&fin, 0u, &dummy, OZ_WAIT_LIMIT);
  } else {
    // ---------------- epilogue: warps 2 .. 2 + OZ_EPI_WARPS - 1
    const int q = warp & 3;                // TMEM lane quarter this warp may access
    const int part = (warp - 2) >> 2;      // column part
    const int row = q * 32 + lane;
    int64_t ngroups = 0;
    bool ok = true;
    df2 acc[OZ_EPI_COLS / 2];   // this group's product, or the sums over the item's groups
    for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const OzItem it = oz_item(a, w);
      const int nsteps = (it.kend - it.kbeg) >> 4;
      const int64_t gm = it.m0 + row, gn0 = it.n0 + part * OZ_EPI_COLS;
      const int nc = (int)min((int64_t)OZ_EPI_COLS, a.Nvalid - gn0);   // this warp's columns (<= 0: none)
      if (E == kOzPairs && w + gridDim.x < nitems) {
        // the next item's C tile streams into L2 while this one is computed:
        // a lane takes one column, 32 rows of 8 bytes
        const OzItem nx = oz_item(a, w + gridDim.x);
        const int64_t pm = nx.m0 + q * 32, pn = nx.n0 + part * OZ_EPI_COLS + lane;
        if (pn < a.Nvalid && pm < a.Mvalid) {
          const float2* pc = a.C + pn * a.ldc + pm;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(pc));
          if (pm + 16 < a.Mvalid) asm volatile("prefetch.global.L2 [%0];" ::"l"(pc + 16));
        }
      }
      if constexpr (E == kOzSums) {
#pragma unroll
        for (int j = 0; j < OZ_EPI_COLS / 2; ++j) acc[j] = {{0ull}, {0ull}};
      }
      for (int t0 = 0; t0 < nsteps; t0 += steps_per_group) {
        // the group's exponents are loaded while its MMAs run
        const int64_t grp = (it.kbeg + t0 * 16) / a.kgroup;
        const int eA = (gm < a.AR) ? a.eA[grp * a.AR + gm] : 0;
        const int eb = (gn0 + lane < a.BR) ? __ldg(a.eB + grp * a.BR + gn0 + lane) : 0;
        int* ebs = s_eb[warp - 2];
        ebs[lane] = eb << 23;
        __syncwarp();
        ok = oz_wait(&acc_full, (uint32_t)(ngroups & 1), &s_fail, a.polls);
        if (!ok) break;
        ++ngroups;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        oz_drain<G, E == kOzSums>(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * OZ_EPI_COLS), ebs, eb, eA, acc);
        // the accumulators are free for the next group (and ebs may be rewritten)
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty);
        if (E != kOzSums && gm < a.Mvalid) {
          if constexpr (E == kOzDoubles) {
            // FP64 storage (a panel's own columns): one FP64 subtraction per element
            double* cp = a.C64 + gn0 * a.ldc + gm;
#pragma unroll
            for (int c16 = 0; c16 < OZ_EPI_COLS; c16 += 16) {
              double cd[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) cd[j] = (c16 + j < nc && !a.c_assign) ? cp[(c16 + j) * a.ldc] : 0.0;
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                if (c16 + j >= nc) continue;
                const float2 h = unpack2(acc[(c16 + j) / 2].h), l = unpack2(acc[(c16 + j) / 2].l);
                const double pv = df_to_double((j & 1) ? f2{h.y, l.y} : f2{h.x, l.x});
                cp[(c16 + j) * a.ldc] = a.c_assign ? pv : cd[j] - pv;
              }
            }
          } else {
            // C -= product, 16 columns per batch of loads
            float2* cp = a.C + gn0 * a.ldc + gm;
#pragma unroll
            for (int c16 = 0; c16 < OZ_EPI_COLS; c16 += 16) {
              float2 cv[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) cv[j] = (c16 + j < nc) ? cp[(c16 + j) * a.ldc] : make_float2(0.0f, 0.0f);
#pragma unroll
              for (int j = 0; j < 16; j += 2) {
                const df2 r = oz_subtract<G>({pack2(cv[j].x, cv[j + 1].x), pack2(cv[j].y, cv[j + 1].y)},
                                             acc[(c16 + j) / 2]);
                const float2 h = unpack2(r.h), l = unpack2(r.l);
                cv[j] = make_float2(h.x, l.x);
                cv[j + 1] = make_float2(h.y, l.y);
              }
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (c16 + j < nc) cp[(c16 + j) * a.ldc] = cv[j];
            }
            // Finished rows become FP64 in a short loop of their own, over what this
            // lane has just stored: the FP64 addition takes its slot of the pipe in
            // every tile where it stands in the loop above, also where it is off.
            if (gm < a.fp64_rows) {
#pragma unroll 1
              for (int j = 0; j < nc; ++j) {
                const float2 v = cp[j * a.ldc];
                *reinterpret_cast<double*>(cp + j * a.ldc) = df_to_double({v.x, v.y});
              }
            }
          }
        }
      }
      if (E == kOzSums && ok) oz_store_sums(a, it, row, part, acc);
    }
  }
  __syncthreads();
  if (s_fail && tid == 0) record_status(a.status, CANDMC_ERR_TIMEOUT);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// Z = Y^T C over K splits, C read as it is stored: a column of C meets the
// tensor cores once (one M tile, b <= 128), so slicing it in its own kernel
// wrote 14 bytes per element that were read back once (450 us at 16384 x 8192
// beside the 605 us of the contraction).  Here twelve warps slice it on the
// way, in two teams of six: team v takes the K16 steps t = v (mod 2) of a group
// and so one stage of the two-stage B ring, a warp 16 columns of them.  (With
// every warp in every step, a step took the 1900 cycles of one warp's chain of
// loads, digits, fence and copies, for 1390 of MMAs.)  The 128 rows of a group
// come into shared memory by asynchronous copies one group ahead, 98 KB, each
// warp its own part, so that only the warp waits for it.  Per group the warps
// find their columns' maxima over their steps' rows and exchange them, then slice
// step after step and ask for the same rows of the next group.  The first step of
// the next group is sliced before the accumulators of the last one are read, so
// the tensor cores go on as soon as they are free.  For the sums, warp w reads TMEM
// lanes 32 (w % 4) .., column part (w - 2) / 4.
constexpr int TN_ASTAGES = 3, TN_BSTAGES = 2;
template <int S>
struct TnCfg {
  static constexpr int A = S * OZ_ABYTES, B = S * OZ_BBYTES;
  static constexpr int RAW = OZ_N * 128 * 8;
  static constexpr int SMEM = TN_ASTAGES * A + TN_BSTAGES * B + RAW + 1024;
};
constexpr int TN_TEAM = OZ_EPI_WARPS / TN_BSTAGES;   // warps of a slicing team
static_assert(OZ_N == 16 * TN_TEAM && 8 % TN_BSTAGES == 0, "two core-matrix row blocks of B per slicing warp");

// asynchronous copies of `bytes` bytes (0 up to 8 or 16), the rest zero
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Where the 16 bytes of rows 2c, 2c + 1 of a warp's column r stand in its 8 x 16
// block (a column takes 128 bytes): moved among the 8 places of the column so that the
// slicing lanes' reads (rows of 4 columns, 2 places apart) fall on different banks.
__device__ __forceinline__ uint32_t raw_place(int r, int c) {
  return (uint32_t)(r * 128 + ((c ^ ((r & 1) | ((r & 2) << 1))) << 4));
}

// the scale exponent of a column whose halves have these maxima (the lo part can
// push |x| just above |hi|'s bound; leave one ulp of room)
__device__ __forceinline__ int tn_exp(float m0, float m1) { return scale_exp(fmaxf(m0, m1) * (1.0f + 1.0e-6f)); }

template <int S>
__global__ void __launch_bounds__(OZ_THREADS, 1) k_oz_tn(OzArgs a) {
  constexpr int G = OzCfg<S>::G;
  using Cfg = TnCfg<S>;
  extern __shared__ __align__(1024) unsigned char oz_smem[];
  __shared__ __align__(8) uint64_t a_full[TN_ASTAGES], a_empty[TN_ASTAGES], b_full[TN_BSTAGES], b_empty[TN_BSTAGES];
  __shared__ __align__(8) uint64_t acc_full, acc_empty, exp_full, fin;
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int s_fail;
  __shared__ float s_mx[2][TN_BSTAGES][OZ_N];      // column maxima by group parity and team
  __shared__ int s_eb[OZ_EPI_WARPS][OZ_EPI_COLS];   // per warp: the exponents of its sums' columns
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  unsigned char* ring = (unsigned char*)(((uintptr_t)oz_smem + 1023) & ~(uintptr_t)1023);
  const int nitems = a.n_nt * a.n_ks;

  if (tid == 0) {
    for (int st = 0; st < TN_ASTAGES; ++st) {
      mbar_init(&a_full[st], 1);
      mbar_init(&a_empty[st], 1);
    }
    for (int st = 0; st < TN_BSTAGES; ++st) {
      mbar_init(&b_full[st], TN_TEAM);
      mbar_init(&b_empty[st], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, OZ_EPI_WARPS);
    mbar_init(&exp_full, OZ_EPI_WARPS);
    mbar_init(&fin, 1);
    s_fail = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_s)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // An A operand of fewer than 128 rows (a narrow Y^T, stored with AR rows)
  // fills only the first AR x 32 bytes of each slice block; the rest of every
  // stage's A blocks is zeroed once here and never written again, so the
  // 128-row MMA reads zeros there.
  if (a.AR < OZ_M) {
    const int abytes = (int)a.AR * 32;
    const int tail = (OZ_ABYTES - abytes) / 16;
    for (int idx = tid; idx < TN_ASTAGES * S * tail; idx += blockDim.x) {
      const int blk = idx / tail, q = idx % tail;
      *reinterpret_cast<uint4*>(ring + (size_t)blk * OZ_ABYTES + abytes +
                                16 * q) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  unsigned char* bring = ring + TN_ASTAGES * Cfg::A;

  if (warp == 0) {
    // ---------------- producer of A: the whole warp walks the stages, one elected lane copies
    const int abytes = (a.AR < OZ_M) ? (int)a.AR * 32 : OZ_ABYTES;
    const int64_t aplane = a.AR * a.Kpad;
    int st = 0, fills = 0;
    uint32_t parity = 1;
    bool ok = true;
    for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const OzItem it = oz_item(a, w);
      const __nv_bfloat16* as = a.As + (int64_t)it.kbeg * a.AR;
      for (int k = it.kbeg; k < it.kend; k += 16, as += a.AR * 16) {
        ok = oz_wait(&a_empty[st], parity, &s_fail, a.polls);
        if (!ok) break;
        ++fills;
        if (elect_one()) {
          mbar_expect_tx(&a_full[st], (unsigned)(S * abytes));
          const uint32_t sa = smem_u32(ring + st * Cfg::A);
#pragma unroll
          for (int sl = 0; sl < S; ++sl) bulk_g2s(sa + sl * OZ_ABYTES, as + sl * aplane, (unsigned)abytes, &a_full[st]);
        }
        __syncwarp();
        if (++st == TN_ASTAGES) {
          st = 0;
          parity ^= 1;
        }
      }
    }
    oz_copies_done(a_full, TN_ASTAGES, fills);
  } else if (warp == 1) {
    // ---------------- MMA issuer: the whole warp walks the stages, one elected lane issues
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_N >> 3) << 17) |
                           ((uint32_t)(OZ_M >> 4) << 24);
    // the rings end below 256 KB: base + offset / 16 stays inside the
    // descriptor's 14-bit address field
    const uint64_t a_desc = make_desc(smem_u32(ring)), b_desc = make_desc(smem_u32(bring));
    static_assert(Cfg::A % 1024 == 0 && Cfg::B % 1024 == 0 && Cfg::SMEM + 2048 < (1 << 18), "stage alignment, range");
    int sa = 0, sb = 0;
    uint32_t a_parity = 0, b_parity = 0, acc_parity = 1;
    bool ok = true;
    for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const OzItem it = oz_item(a, w);
      for (int k = it.kbeg; k < it.kend && ok; k += 128) {
        // the previous group's accumulators have been read
        ok = oz_wait(&acc_empty, acc_parity, &s_fail, a.polls);
        acc_parity ^= 1;
        for (int t = 0; t < 8 && ok; ++t) {
          ok = oz_wait(&a_full[sa], a_parity, &s_fail, a.polls) && oz_wait(&b_full[sb], b_parity, &s_fail, a.polls);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          oz_issue_step<S, G>(tmem, a_desc + (uint64_t)(sa * (Cfg::A >> 4)), b_desc + (uint64_t)(sb * (Cfg::B >> 4)),
                              idesc, t > 0 ? 1u : 0u);
          umma_commit(&b_empty[sb]);   // the stages are free once these MMAs have read them
          umma_commit(&a_empty[sa]);
          if (++sa == TN_ASTAGES) {
            sa = 0;
            a_parity ^= 1;
          }
          if (++sb == TN_BSTAGES) {
            sb = 0;
            b_parity ^= 1;
          }
        }
        if (ok) umma_commit(&acc_full);
      }
    }
    // every MMA this warp issued has completed before TMEM is released
    umma_commit(&fin);
    volatile int dummy = 0;
    oz_wait(&fin, 0u, &dummy, OZ_WAIT_LIMIT);
  } else {
    // ---------------- slicing of C and sums: warps 2 .. 2 + OZ_EPI_WARPS - 1
    const int cw = warp - 2;
    const int team = cw / TN_TEAM, c0 = (cw % TN_TEAM) * 16;   // steps team, team + 2, ..; columns c0 .. c0 + 15
    const int q = warp & 3;                // TMEM lane quarter this warp may access
    const int part = cw >> 2;              // column part of the sums
    const int row = q * 32 + lane;
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * OZ_EPI_COLS);
    unsigned char* raw = bring + TN_BSTAGES * Cfg::B + cw * 8192;   // 4 K16 blocks of 16 columns x 16 rows
    const double* C = reinterpret_cast<const double*>(a.C);   // a float pair takes 8 bytes
    // Asynchronous copies of this warp's part of a group, block after block: a lane
    // takes 16 bytes (2 rows) of every fourth column where C's columns are aligned to
    // that, else 8 bytes (1 row) of every second.  load_from sets the lane's first element.
    const bool wide = ((a.ldc | (int64_t)(reinterpret_cast<uintptr_t>(C) >> 3)) & 1) == 0;
    const int lrow = wide ? 2 * (lane & 7) : (lane & 15), lcol = wide ? lane >> 3 : lane >> 4;
    const uint32_t ldst = smem_u32(raw);
    const double* lp = C;
    int lleft = 0, lcols = 0;   // rows and columns from the lane's first element to the matrix' end
    auto load_from = [&](int64_t n0, int k) {
      const int64_t n = n0 + c0 + lcol;
      lp = C + n * a.ldc + k + team * 16 + lrow;
      lleft = (int)a.Kvalid - k - team * 16 - lrow;
      lcols = (int)min(a.Nvalid - n, (int64_t)16);
    };
    auto load_block = [&](int u) {   // the warp's u-th step of the group
      const double* p = lp + u * 32;
      const int left = lleft - u * 32;
      if (wide) {
        const int bytes = min(max(left, 0), 2) * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int b = 4 * i < lcols ? bytes : 0;
          cp_async16(ldst + u * 2048 + raw_place(lcol + 4 * i, lrow >> 1), b ? p + i * 4 * a.ldc : C, b);
        }
      } else {
        const int bytes = left > 0 ? 8 : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int b = 2 * i < lcols ? bytes : 0;
          cp_async8(ldst + u * 2048 + raw_place(lcol + 2 * i, lrow >> 1) + (lane & 1) * 8, b ? p + i * 2 * a.ldc : C, b);
        }
      }
    };
    // lane's part of a block: columns r and r + 8, rows kr .. kr + 3
    const int r = (lane & 15) >> 1, kr = (lane >> 4) * 8 + (lane & 1) * 4;
    const uint32_t place0 = raw_place(r, kr >> 1), place1 = raw_place(r, (kr >> 1) + 1);
    // maxima of the lane's columns over a block's rows, once they have arrived
    float mx[2] = {0.0f, 0.0f};
    auto scan_block = [&](int u) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float4 x = *reinterpret_cast<const float4*>(raw + u * 2048 + (c >> 1) * 1024 + ((c & 1) ? place1 : place0));
        mx[c >> 1] = fmaxf(mx[c >> 1], fmaxf(fabsf(x.x), fabsf(x.z)));
      }
    };
    df2 acc[OZ_EPI_COLS / 2];   // sums over the item's K range
#pragma unroll
    for (int j = 0; j < OZ_EPI_COLS / 2; ++j) acc[j] = {{0ull}, {0ull}};

    // The accumulators of the group at row k of item it are read and added up;
    // after its last group the item's sums are written.
    uint32_t drained = 0;
    auto drain = [&](const OzItem& it, int k, int eA) -> bool {
      const uint32_t par = drained & 1;
      const int c = part * OZ_EPI_COLS + lane;
      const int eb = tn_exp(s_mx[par][0][c], s_mx[par][1][c]);
      s_eb[cw][lane] = eb << 23;
      if (!oz_wait(&acc_full, par, &s_fail, a.polls)) return false;
      ++drained;
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      oz_drain<G, true>(taddr, s_eb[cw], eb, eA, acc);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty);
      if (k + 128 < it.kend) return true;
      oz_store_sums(a, it, row, part, acc);
#pragma unroll
      for (int j = 0; j < OZ_EPI_COLS / 2; ++j) acc[j] = {{0ull}, {0ull}};
      return true;
    };

    OzItem it = oz_item(a, blockIdx.x), last_it = it;
    int w = blockIdx.x, k = it.kbeg, last_k = -1, last_eA = 0;
    uint32_t b_parity = 1, group = 0;
    bool ok = true;
    load_from(it.n0, k);
#pragma unroll 1
    for (int u = 0; u < 4; ++u) load_block(u);
    bool have = true;   // a group to slice; the last pass only reads the last group's sums
    while (true) {
      const int eA = (have && row < a.AR) ? a.eA[(int64_t)(k >> 7) * a.AR + row] : 0;
      OzItem nit = it;
      int nw = w, nk = k + 128;
      bool more = have;
      int e[2] = {0, 0};
      if (have) {
      // the last of this warp's rows of the group have arrived (the first group: all)
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
#pragma unroll 1
      for (int u = group ? 3 : 0; u < 4; ++u) scan_block(u);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 16));
        if ((lane & 17) == 0) s_mx[group & 1][team][c0 + r + 8 * h] = mx[h];
        mx[h] = 0.0f;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&exp_full);
      // the group after this one
      if (nk >= it.kend) {
        nw = w + gridDim.x;
        more = nw < nitems;
        if (more) {
          nit = oz_item(a, nw);
          nk = nit.kbeg;
        }
      }
      load_from(nit.n0, nk);
      ok = oz_wait(&exp_full, group & 1, &s_fail, a.polls);
      if (!ok) break;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        e[h] = tn_exp(s_mx[group & 1][0][c0 + r + 8 * h], s_mx[group & 1][1][c0 + r + 8 * h]);
      }
      const bool tiny = __any_sync(0xffffffffu, min(e[0], e[1]) < -119);
      // Team 0 prepares the first step before it reads the last group's sums; the second
      // step's stage is free only with the last group's last MMA, so team 1 reads them first.
#pragma unroll 1
      for (int u = 0; u < 4; ++u) {
        if (u == 1 - team && last_k >= 0) {
          ok = drain(last_it, last_k, last_eA);
          if (!ok) break;
        }
        if (!have) continue;
        unsigned char* sd = bring + team * Cfg::B + c0 * 32 + lane * 8;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 x0 = *reinterpret_cast<const float4*>(raw + u * 2048 + h * 1024 + place0);
          const float4 x1 = *reinterpret_cast<const float4*>(raw + u * 2048 + h * 1024 + place1);
          // times 2^(8 - e): two normal factors, the second one 1 unless e < -119
          const int k1 = min(8 - e[h], 127);
          const float f1 = pow2f(k1);
          f2x2 v[4] = {pack2(x0.x, x0.z), pack2(x0.y, x0.w), pack2(x1.x, x1.z), pack2(x1.y, x1.w)};
          if (tiny) {
            const float f2v = pow2f(8 - e[h] - k1);
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = mul2(v[c], pack2(f2v, f2v));
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) v[c] = mul2(v[c], pack2(f1, f1));
          uint32_t d[S][2];
          slice_digits<S>(v[0], v[1], [&](int i, f2x2 y) { d[i][0] = to_bf16x2(y); });
          slice_digits<S>(v[2], v[3], [&](int i, f2x2 y) { d[i][1] = to_bf16x2(y); });
          if (h == 0) {
            // while the stage is in use: the block asked for one step ago
            if (u > 0 && more) {
              asm volatile("cp.async.wait_all;" ::: "memory");
              __syncwarp();
              scan_block(u - 1);
            }
            ok = oz_wait(&b_empty[team], b_parity, &s_fail, a.polls);
            if (!ok) break;
          }
#pragma unroll
          for (int i = 0; i < S; ++i)
            *reinterpret_cast<uint2*>(sd + h * 256 + i * OZ_BBYTES) = make_uint2(d[i][0], d[i][1]);
        }
        if (!ok) break;
        b_parity ^= 1;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_full[team]);
        if (more) load_block(u);
      }
      last_it = it;
      last_k = k;
      last_eA = eA;
      ++group;
      if (!ok || !have) break;
      have = more;
      it = nit;
      w = nw;
      k = nk;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  if (s_fail && tid == 0) record_status(a.status, CANDMC_ERR_TIMEOUT);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// ------------------------------------------------------------------ conversions and reduction
// FP64 <-> df64 in place, m x n: a CTA takes kCvtRows rows of a column (no
// division per element), four loads in flight per thread.  Bound by memory (16 B
// per element): 8192 x 4096 in 241 / 182 us with FP64-pipe conversions.
constexpr int kCvtRows = 1024;
template <bool TO>
__global__ void __launch_bounds__(256) k_cvt_df64(double* X, int64_t ld, int64_t m, int64_t n) {
  const int64_t r0 = (int64_t)blockIdx.x * kCvtRows + threadIdx.x;
  for (int64_t j = blockIdx.y; j < n; j += gridDim.y) {
    double* p = X + j * ld;
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = r0 + 256 * u < m ? p[r0 + 256 * u] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      double w;
      if (TO) {
        const f2 t = df_from_double(v[u]);
        w = __hiloint2double(__float_as_int(t.l), __float_as_int(t.h));   // float2 {h, l}
      } else {
        w = df_to_double({__int_as_float(__double2loint(v[u])), __int_as_float(__double2hiint(v[u]))});
      }
      if (r0 + 256 * u < m) p[r0 + 256 * u] = w;
    }
  }
}

// Z (nb x n, FP64, ld nb) = sum over splits of the df64 partials [split][n][AR],
// added in a fixed order.  Eight partials are loaded before they are added, so
// that a narrow update's many splits (up to one per 128 rows) cost a few memory
// latencies per output; and with W > 1 each of W warps takes 1 / W of the splits
// of a CTA's 256 / W outputs, added up in shared memory (W = 8 from 16 splits:
// 64 splits of 32 x 32 outputs took 12 us with one thread per output).
template <int W>
__global__ void __launch_bounds__(256) k_oz_sum_partials(const float2* part, int nsplit, int64_t AR, int nb,
                                                         int64_t n, double* Z) {
  constexpr int OUT = 256 / W;
  __shared__ float2 sums[W][OUT];
  const int o = threadIdx.x % OUT, w = threadIdx.x / OUT;
  const int64_t idx = (int64_t)blockIdx.x * OUT + o;
  const bool valid = idx < (int64_t)nb * n;
  const int64_t i = idx % nb, j = idx / nb, stride = n * AR;
  const float2* p = part + j * AR + i;
  const int per = (nsplit + W - 1) / W, end = min(nsplit, (w + 1) * per);
  f2 s = {0.0f, 0.0f};
  for (int sp = w * per; valid && sp < end; sp += 8) {
    float2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = sp + u < end ? p[(int64_t)(sp + u) * stride] : make_float2(0.0f, 0.0f);
#pragma unroll
    for (int u = 0; u < 8; ++u) s = df_add(s, {v[u].x, v[u].y});
  }
  if (W > 1) {
    sums[w][o] = make_float2(s.h, s.l);
    __syncthreads();
    if (w) return;
    for (int u = 1; u < W; ++u) s = df_add(s, {sums[u][o].x, sums[u][o].y});
  }
  if (valid) Z[j * nb + i] = df_to_double(s);
}

// ------------------------------------------------------------------ host side
static inline int64_t rup(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

static int num_sms_oz() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

int to_df64(double* X, int64_t ld, int64_t m, int64_t n, cudaStream_t s) {
  if (m <= 0 || n <= 0) return CANDMC_OK;
  ProfScope ps(CANDMC_KCLASS_OZ_SLICE, 16.0 * m * n, s);
  k_cvt_df64<true><<<dim3((unsigned)((m + kCvtRows - 1) / kCvtRows), (unsigned)std::min<int64_t>(n, 65535)), 256, 0, s>>>(X, ld, m, n);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

int from_df64(double* X, int64_t ld, int64_t m, int64_t n, cudaStream_t s) {
  if (m <= 0 || n <= 0) return CANDMC_OK;
  ProfScope ps(CANDMC_KCLASS_OZ_SLICE, 16.0 * m * n, s);
  k_cvt_df64<false><<<dim3((unsigned)((m + kCvtRows - 1) / kCvtRows), (unsigned)std::min<int64_t>(n, 65535)), 256, 0, s>>>(X, ld, m, n);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

// One launch over the operands of `jobs`.
template <int S>
static int launch_slices(std::initializer_list<SliceJob> jobs, cudaStream_t s) {
  SliceJobs a{};
  unsigned blocks = 0;
  double bytes = 0.0;
  int i = 0;
  for (const SliceJob& j : jobs) {
    a.job[i] = j;
    blocks += j.out ? j.blocks() : 0;   // a job without an output is none
    a.end[i++] = blocks;
    if (j.out) bytes += 8.0 * j.Nvalid * j.Kvalid + 2.0 * S * j.Rpad * j.Kpad;
  }
  for (; i < 3; ++i) a.end[i] = blocks;
  ProfScope ps(CANDMC_KCLASS_OZ_SLICE, bytes, s);
  k_slice<S><<<blocks, 256, 0, s>>>(a);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

int g_oz_reserve_sms = 32;
thread_local int t_oz_cap = 0;

// one persistent CTA per SM at most (fewer under a cap), each taking every
// gridDim-th work item
static int64_t oz_ctas() {
  const int64_t sms = num_sms_oz();
  return (t_oz_cap > 0 && t_oz_cap < sms) ? t_oz_cap : sms;
}

// K groups of 128 rows per work item of Y^T C, for `groups` of them and ntiles
// column tiles.  The CTAs take the items in turn, so the time is that of the
// CTA with the most: rounds x (groups per item + what an item costs besides).
// An item's partial tile, written once and read once by the reduction, takes
// about 0.8 of a group's time.  Two rounds of equal items, whatever their
// number came to, left 16384 x 8192 (86 tiles) at 96 groups per CTA, where
// the mean is 72.4; this rule gives 76.
static int64_t oz_groups_per_item(int64_t groups, int64_t ntiles) {
  const int64_t ctas = oz_ctas();
  int64_t best = groups;
  double best_cost = 1e300;
  for (int64_t ks = 1; ks <= groups && (ks == 1 || ntiles * (ks - 1) < 8 * ctas); ++ks) {
    const int64_t per = (groups + ks - 1) / ks;
    const int64_t items = ntiles * ((groups + per - 1) / per);
    const double cost = (double)((items + ctas - 1) / ctas) * ((double)per + 0.8);
    if (cost < best_cost) {
      best_cost = cost;
      best = per;
    }
  }
  return best;
}
// Dynamic shared memory above the default limit, allowed once per kernel.
template <class K>
static int allow_smem(K kernel, int bytes, std::atomic<bool>& done) {
  if (done) return CANDMC_OK;
  CANDMC_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  done = true;
  return CANDMC_OK;
}

template <int S, OzEpilogue E>
static int launch_oz_mma(OzArgs a, int64_t gm, int64_t gn, int64_t gk, int cls, double flops, cudaStream_t s) {
  static std::atomic<bool> attr{false};
  CANDMC_RET(allow_smem(k_oz_mma<S, E>, OzCfg<S>::SMEM, attr));
  a.polls = g_oz_polls;
  a.n_mt = (int)gm;
  a.n_nt = (int)gn;
  a.n_ks = (int)gk;
  ProfScope ps(cls, flops, s);
  k_oz_mma<S, E><<<(unsigned)std::min<int64_t>(gm * gn * gk, oz_ctas()), OZ_THREADS, OzCfg<S>::SMEM, s>>>(a);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

template <int S>
static int launch_oz_tn(OzArgs a, int64_t gn, int64_t gk, int cls, double flops, cudaStream_t s) {
  static std::atomic<bool> attr{false};
  CANDMC_RET(allow_smem(k_oz_tn<S>, TnCfg<S>::SMEM, attr));
  a.polls = g_oz_polls;
  a.n_mt = 1;
  a.n_nt = (int)gn;
  a.n_ks = (int)gk;
  ProfScope ps(cls, flops, s);
  k_oz_tn<S><<<(unsigned)std::min<int64_t>(gn * gk, oz_ctas()), OZ_THREADS, TnCfg<S>::SMEM, s>>>(a);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

// Z (nb x n, FP64, ld nb) = Y^T C with S-slice contractions: Y (m x nb) and C
// (m x n) read through their slice sources; split-K partials summed in df64.
template <int S>
static int oz_tn(const SliceSrc& ysrc, const SliceSrc& csrc, int64_t m, int nb, int64_t n, double* Z,
                 int* status, cudaStream_t s, int cls, const SliceJob& also = SliceJob{}) {
  const int64_t KG = 128;                       // K rows per exact accumulation
  // A-op = Y^T (rows = Householder index, K = m), B-op = C (rows = columns)
  const int64_t Kp1 = rup(m, KG);
  // the A operand keeps only its nb rows (rounded to a core matrix of 8):
  // the kernel zero-fills the rest of the 128-row tile in shared memory
  const int64_t AR1 = rup(nb, 8), ntiles = (n + OZ_N - 1) / OZ_N;
  DevBuf ya, ea, cb, eb, part;
  CANDMC_RET(ya.alloc(sizeof(__nv_bfloat16) * S * AR1 * Kp1, s));
  CANDMC_RET(ea.alloc(sizeof(int) * (Kp1 / KG) * AR1, s));
  auto* yas = static_cast<__nv_bfloat16*>(ya.p);
  const SliceJob yjob{ysrc, 0, m, nb, AR1, Kp1, (int)KG, yas, static_cast<int*>(ea.p)};
  const int64_t kper = KG * oz_groups_per_item(Kp1 / KG, ntiles);
  const int64_t ksplit = (Kp1 + kper - 1) / kper;
  CANDMC_RET(part.alloc(sizeof(float2) * ksplit * n * AR1, s));
  OzArgs g1{};
  g1.As = yas; g1.AR = AR1; g1.Kpad = (int)Kp1; g1.k_per_cta = (int)kper;
  g1.kgroup = (int)KG; g1.eA = static_cast<int*>(ea.p); g1.part = static_cast<float2*>(part.p);
  g1.Mvalid = nb; g1.Nvalid = n; g1.Kvalid = m; g1.status = status;
  const double flops = 2.0 * nb * n * m;
  // Float pairs are sliced on their way through the contraction.  FP64 columns (a
  // panel's own, few column tiles) are sliced by k_slice first: splitting a double
  // by its bits takes more issue slots than the twelve warps have beside the MMAs
  // (the half-panel update of 16384 x 32: 44 us fused, 33 in two kernels).
  if (csrc.df) {
    g1.C = const_cast<float2*>(csrc.df);
    g1.ldc = csrc.ld;
    CANDMC_RET(launch_slices<S>({yjob, also}, s));
    CANDMC_RET(launch_oz_tn<S>(g1, ntiles, ksplit, cls, flops, s));
  } else {
    const int64_t BR1 = ntiles * OZ_N;
    CANDMC_RET(cb.alloc(sizeof(__nv_bfloat16) * S * BR1 * Kp1, s));
    CANDMC_RET(eb.alloc(sizeof(int) * (Kp1 / KG) * BR1, s));
    g1.Bs = static_cast<__nv_bfloat16*>(cb.p); g1.BR = BR1; g1.eB = static_cast<int*>(eb.p);
    const SliceJob cjob{csrc, 0, m, n, BR1, Kp1, (int)KG, static_cast<__nv_bfloat16*>(cb.p), static_cast<int*>(eb.p)};
    CANDMC_RET(launch_slices<S>({yjob, cjob, also}, s));
    CANDMC_RET((launch_oz_mma<S, kOzSums>(g1, 1, ntiles, ksplit, cls, flops, s)));
  }
  ProfScope ps(CANDMC_KCLASS_REDUCE, 8.0 * ksplit * n * AR1, s);
  const int64_t outs = (int64_t)nb * n;
  const auto* pp = static_cast<const float2*>(part.p);
  if (ksplit >= 16)
    k_oz_sum_partials<8><<<(unsigned)((outs + 31) / 32), 256, 0, s>>>(pp, (int)ksplit, AR1, nb, n, Z);
  else
    k_oz_sum_partials<1><<<(unsigned)((outs + 255) / 256), 256, 0, s>>>(pp, (int)ksplit, AR1, nb, n, Z);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

// Zt (nb x n, FP64, ld nb) = Top (nb x nb) * Z (nb x n, FP64, ld nb) with the
// S-slice contraction: Top is the A operand (sliced from its stored matrix,
// transposed or not), Z the B operand, and the epilogue stores the
// product into Zt instead of subtracting it.
template <int S>
static int oz_top_times(MatRef Top, int nb, const double* Z, int64_t n, double* Zt, int* status,
                        cudaStream_t s, int cls) {
  const int64_t Kp = rup(nb, 16), BR = rup(n, OZ_N);
  DevBuf ta, et, zb, ez;
  CANDMC_RET(ta.alloc(sizeof(__nv_bfloat16) * S * OZ_M * Kp, s));
  CANDMC_RET(et.alloc(sizeof(int) * OZ_M, s));
  CANDMC_RET(zb.alloc(sizeof(__nv_bfloat16) * S * BR * Kp, s));
  CANDMC_RET(ez.alloc(sizeof(int) * BR, s));
  auto* tas = static_cast<__nv_bfloat16*>(ta.p);
  auto* zbs = static_cast<__nv_bfloat16*>(zb.p);
  const SliceSrc tsrc{Top.p, nullptr, Top.ld, Top.mask, Top.off};
  // A operand element (i, k) = Top(i, k): X[k, i] of a transposed reference
  // (a column of X per operand row), X[i, k] otherwise (a row of X)
  const SliceJob tjob{tsrc, Top.trans ? 0 : 1, nb, nb, OZ_M, Kp, (int)Kp, tas, static_cast<int*>(et.p)};
  const SliceJob zjob{SliceSrc{Z, nullptr, nb, kDense, 0}, 0, nb, n, BR, Kp, (int)Kp, zbs, static_cast<int*>(ez.p)};
  CANDMC_RET(launch_slices<S>({tjob, zjob}, s));
  OzArgs g{};
  g.As = tas; g.AR = OZ_M; g.Bs = zbs; g.BR = BR;
  g.Kpad = g.k_per_cta = g.kgroup = (int)Kp;
  g.eA = static_cast<int*>(et.p); g.eB = static_cast<int*>(ez.p);
  g.C = reinterpret_cast<float2*>(Zt); g.C64 = Zt; g.ldc = nb;
  g.Mvalid = nb; g.Nvalid = n; g.fp64_rows = 0; g.status = status;
  g.c_assign = 1;
  return launch_oz_mma<S, kOzDoubles>(g, 1, BR / OZ_N, 1, cls, 2.0 * nb * nb * n, s);
}

// Width from which the operator product T^T Z of an update runs on the
// tensor cores (below it, the FP64 small-matrix kernel is quicker).
constexpr int64_t kOzTopMinCols = 1024;

// The trailing update with S-slice contractions: C <- C - Y (Top (Y^T C)).
// C (m x n, ld ldc) holds df64 pairs; rows < fp64_rows of C are written back
// as FP64 (finished R rows).  With c_fp64, C is FP64 storage instead (read and
// written as FP64).  Y: unit-lower m x nb (read from a Y\R buffer, FP64),
// Top: the nb x nb operator applied to Y^T C.  cls_tn / cls_nn: the kernel
// classes the two contractions are counted under.
template <int S>
static int apply_qt_slices(const double* Y, int64_t ldy, int ymask, int64_t m, int nb, MatRef Top,
                           double* C, int64_t ldc, int64_t n, int64_t fp64_rows, int* status,
                           cudaStream_t s, bool c_fp64, int cls_tn, int cls_nn) {
  if (m <= 0 || n <= 0) return CANDMC_OK;
  if (nb > OZ_M) return set_error(CANDMC_ERR_ARG, "ozaki form needs b <= 128");
  // ---- GEMM1: Z = Y^T C
  SliceSrc ysrc{Y, nullptr, ldy, ymask, 0};
  SliceSrc csrc = c_fp64 ? SliceSrc{C, nullptr, ldc, kDense, 0}
                         : SliceSrc{nullptr, reinterpret_cast<const float2*>(C), ldc, kDense, 0};
  DevBuf z, zt;
  CANDMC_RET(z.alloc(sizeof(double) * nb * n, s));
  // Y as the A operand of GEMM2 (rows = m, K = nb) is sliced in the same launch
  const int64_t Kp2 = rup(nb, 16);
  const int64_t AR2 = rup(m, OZ_M), BR2 = rup(n, OZ_N);
  DevBuf y2, ey2, z2, ez2;
  CANDMC_RET(y2.alloc(sizeof(__nv_bfloat16) * S * AR2 * Kp2, s));
  CANDMC_RET(ey2.alloc(sizeof(int) * AR2, s));
  const SliceJob y2job{ysrc, 1, nb, m, AR2, Kp2, (int)Kp2, static_cast<__nv_bfloat16*>(y2.p), static_cast<int*>(ey2.p)};
  CANDMC_RET(oz_tn<S>(ysrc, csrc, m, nb, n, z.d(), status, s, cls_tn, y2job));
  // ---- Z' = T^T * Z   (FP64 storage, nb x n); counted, as on the FP64 pipe,
  // under the small-product class, apart from the two contractions with Y
  CANDMC_RET(zt.alloc(sizeof(double) * nb * n, s));
  if (n >= kOzTopMinCols)
    CANDMC_RET(oz_top_times<S>(Top, nb, z.d(), n, zt.d(), status, s, CANDMC_KCLASS_SMALL));
  else
    CANDMC_RET(small_gemm(nb, n, nb, 1.0, Top, mref(z.d(), nb), 0.0, zt.d(), nb, s));
  // ---- GEMM2: C -= Y * Z'.  A-op = Y (rows = m, K = nb), B-op = Z'^T (rows = columns, K = nb)
  CANDMC_RET(z2.alloc(sizeof(__nv_bfloat16) * S * BR2 * Kp2, s));
  CANDMC_RET(ez2.alloc(sizeof(int) * BR2, s));
  CANDMC_RET(launch_slices<S>({SliceJob{SliceSrc{zt.d(), nullptr, nb, kDense, 0}, 0, nb, n, BR2, Kp2, (int)Kp2,
                                        static_cast<__nv_bfloat16*>(z2.p), static_cast<int*>(ez2.p)}}, s));
  OzArgs g2{};
  g2.As = static_cast<__nv_bfloat16*>(y2.p); g2.AR = AR2;
  g2.Bs = static_cast<__nv_bfloat16*>(z2.p); g2.BR = BR2;
  g2.Kpad = g2.k_per_cta = g2.kgroup = (int)Kp2;
  g2.eA = static_cast<int*>(ey2.p); g2.eB = static_cast<int*>(ez2.p);
  g2.C = reinterpret_cast<float2*>(C); g2.C64 = C; g2.ldc = ldc;
  g2.Mvalid = m; g2.Nvalid = n; g2.fp64_rows = fp64_rows; g2.status = status;
  const double flops = 2.0 * m * n * nb;
  if (c_fp64) return launch_oz_mma<S, kOzDoubles>(g2, AR2 / OZ_M, BR2 / OZ_N, 1, cls_nn, flops, s);
  return launch_oz_mma<S, kOzPairs>(g2, AR2 / OZ_M, BR2 / OZ_N, 1, cls_nn, flops, s);
}

// The emulated-FP64 form: 7 slices, 28 slice products per K16 step.
int apply_qt_ozaki(const double* Y, int64_t ldy, int ymask, int64_t m, int nb, MatRef Top,
                   double* C, int64_t ldc, int64_t n, int64_t fp64_rows, int* status,
                   cudaStream_t s, bool c_fp64) {
  // a panel's own half-panel updates (FP64 storage) are counted apart from
  // the trailing-matrix contractions
  return apply_qt_slices<OZ_S>(Y, ldy, ymask, m, nb, Top, C, ldc, n, fp64_rows, status, s, c_fp64,
                               c_fp64 ? CANDMC_KCLASS_OZ_PANEL : CANDMC_KCLASS_OZ_TN,
                               c_fp64 ? CANDMC_KCLASS_OZ_PANEL : CANDMC_KCLASS_OZ_NN);
}

// The FP32 form on the same tensor-core path: 3 BF16 slices (24 bits under
// each scale group's exponent, FP32-class accuracy), 6 slice products per K16
// step in 3 accumulator groups, summed in FP32.  C keeps the df64 slots of
// the emulated form, but the epilogue updates it in FP32 arithmetic (its low
// word becomes zero), so the read-modify-write costs one FP32 operation per
// element instead of a df64 addition.
int apply_qt_f32(const double* Y, int64_t ldy, int ymask, int64_t m, int nb, MatRef Top, double* C,
                 int64_t ldc, int64_t n, int64_t fp64_rows, int* status, cudaStream_t s) {
  return apply_qt_slices<OZ_S32>(Y, ldy, ymask, m, nb, Top, C, ldc, n, fp64_rows, status, s, false,
                                 CANDMC_KCLASS_F32, CANDMC_KCLASS_F32);
}

// G (nb x n, FP64, ld nb) = Y^T C for FP64 Y (m x nb, mask ymask) and C
// (m x n, mask cmask) in emulated FP64: the Gram product of a panel's
// recursive T merge.
int gram_ozaki(const double* Y, int64_t ldy, int ymask, const double* C, int64_t ldc, int cmask, int64_t m,
               int nb, int64_t n, double* G, int* status, cudaStream_t s) {
  if (m <= 0 || n <= 0 || nb <= 0) return CANDMC_OK;
  if (nb > OZ_M) return set_error(CANDMC_ERR_ARG, "gram_ozaki needs nb <= 128");
  return oz_tn<OZ_S>(SliceSrc{Y, nullptr, ldy, ymask, 0}, SliceSrc{C, nullptr, ldc, cmask, 0}, m, nb, n, G,
                     status, s, CANDMC_KCLASS_OZ_PANEL);
}

}  // namespace candmc
