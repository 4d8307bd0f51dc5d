// FP64 contractions of the CAQR trailing update and the small b x b products.
//
// Reference: upd_A (alg/QR/qr_2d/qr_2d.cxx:224-282) computes Z = Y^T*A with
// dgemm (:259), all-reduces Z over the process column (:265), applies T^T by
// dtrsm with T^-T (:271) and finishes with A -= Y*Z by dgemm (:275).  On one
// GPU the all-reduce becomes a deterministic split-K reduction: each CTA of
// gemm_tn owns a slice of rows and writes a partial Z, and reduce_apply sums
// the partials in a fixed order and multiplies by T^T in the same pass.
//
// GB300 note: FP64 runs at ~1.2 TFLOP/s chip-wide (a warp-wide FP64 instruction
// takes 65 cycles of its sub-partition), so these kernels are bound by the
// number of FP64 instructions: tiles that fit the product's odd widths count
// for more than operand reuse.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace candmc {

// ---- products of up to kSmallProduct multiplications: out(i, j) = sum_{k in
// [k0, k1)} opA(i, k) * opB(k, j), a 16 x 16 tile per CTA, one output a thread.
// Many small CTAs spread such a product over the SMs and run little code once
// (1500 x 32 x 32: 9 us against 11 and 20 in the two kernels below; 8192 x 32 x
// 32: 20 against 27 and 40); from 8192 x 64 x 64 on the others are ahead.
// mode 0: store into out + split * split_stride (partials), ld ldo.
// mode 1: out(i, j) -= result (out is the trailing matrix itself).
constexpr int TK = 16;
static_assert(kThreads == 16 * TK, "one tile element a thread");
constexpr int64_t kSmallProduct = 20000000;

__global__ void __launch_bounds__(kThreads)
k_gemm_f64(MatRef A, MatRef B, int64_t M, int64_t N, int64_t K, int64_t kchunk, double* out,
           int64_t ldo, int64_t split_stride, int mode) {
  constexpr int TM = 16, TN = 16;
  __shared__ double sA[TK][TM + 1];
  __shared__ double sB[TK][TN + 1];
  const int tid = threadIdx.x;
  const int ti = tid % 16, tj = tid / 16;
  const int64_t i0 = (int64_t)blockIdx.x * TM, j0 = (int64_t)blockIdx.y * TN;
  const int64_t k0 = (int64_t)blockIdx.z * kchunk;
  const int64_t k1 = (k0 + kchunk < K) ? k0 + kchunk : K;
  double acc = 0.0;
  for (int64_t kb = k0; kb < k1; kb += TK) {
    // one element of each tile a thread, coalesced along the stored row index
    {
      int ii, kk;
      if (A.trans) { kk = tid % TK; ii = tid / TK; } else { ii = tid % TM; kk = tid / TM; }
      const int64_t gi = i0 + ii, gk = kb + kk;
      sA[kk][ii] = (gi < M && gk < k1) ? mat_at(A, gi, gk) : 0.0;
    }
    {
      int jj, kk;
      if (B.trans) { jj = tid % TN; kk = tid / TN; } else { kk = tid % TK; jj = tid / TK; }
      const int64_t gj = j0 + jj, gk = kb + kk;
      sB[kk][jj] = (gj < N && gk < k1) ? mat_at(B, gk, gj) : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) acc = fma(sA[kk][ti], sB[kk][tj], acc);
    __syncthreads();
  }
  const int64_t gi = i0 + ti, gj = j0 + tj;
  if (gi >= M || gj >= N) return;
  double* o = out + (mode == 0 ? (int64_t)blockIdx.z * split_stride : 0) + gj * ldo + gi;
  if (mode == 0) *o = acc;
  else *o -= acc;
}

// An operand as element (i, j) = p[i si + j sj] with its mask as what to keep by
// the sign of d = +-(i - j) - off: mat_at with its transposition and mask worked
// out once, in a dozen instructions an element.  These kernels are short, and
// code that runs once costs about 30 cycles an instruction to fetch: with
// mat_at's switch inlined per load, a product of 8192 x 32 x 32 took 45 us.
struct View {
  const double* p;
  int64_t si, sj, off;
  int sgn;
  bool pos, zero, neg, unit;   // keep d > 0, d == 0, d < 0; d == 0 reads as one
};

__device__ __forceinline__ View make_view(const MatRef& X) {
  View v;
  v.p = X.p;
  v.si = X.trans ? X.ld : 1;
  v.sj = X.trans ? 1 : X.ld;
  v.off = X.off;
  v.sgn = X.trans ? -1 : 1;
  v.pos = X.mask != kUpper;
  v.neg = X.mask == kUpper || X.mask == kDense;
  v.unit = X.mask == kUnitLower;
  v.zero = !v.unit;
  return v;
}

__device__ __forceinline__ double view_at(const View& v, int64_t i, int64_t j, bool in) {
  const int64_t d = v.sgn * (i - j) - v.off;
  const bool keep = in && (d > 0 ? v.pos : d < 0 ? v.neg : v.zero);
  const double x = keep ? v.p[i * v.si + j * v.sj] : 0.0;
  return (in && d == 0 && v.unit) ? 1.0 : x;
}

// ---- Y^T C, split over rows
//
// out + z split_stride, (nb x n, ld nb) = sum over the rows of chunk z of
// Y(k, i) C(k, j).  A CTA takes up to 64 x (16 CG) outputs in 8 x 4 lane blocks
// (lane l: row l % 8, column l / 8 of a block), so a product 50 wide pads to 56
// x 52 and not to 64 x 64.  CG warps share the columns (blocks g, g + CG, ..,
// at most four each), the 8 / CG groups of them the rows of a stage, 32 at a
// time through shared memory with the next stage's loads in flight.  The
// groups' sums meet in shared memory at the end.
constexpr int kTnK = 32;              // rows per stage
constexpr int kTnLd = kTnK + 1;

// The sizes are compiled in: a guarded FP64 instruction is predicated, and one
// whose predicate is off for the whole warp still takes its 65 cycles.
template <int NU, int NV, int KG>
__device__ __forceinline__ void tn_stage(const double* sA, const double* sB, int kg, int kn, int bstep,
                                         double (&acc)[8][4]) {
#pragma unroll 1
  for (int k = kg; k < kn; k += KG) {
    double x[NU], y[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) y[v] = sB[v * bstep + k];
#pragma unroll
    for (int u = 0; u < NU; ++u) x[u] = sA[8 * u * kTnLd + k];
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[u][v] = fma(x[u], y[v], acc[u][v]);
  }
}

template <int NV, int KG>
__device__ __forceinline__ void tn_rows(int nu, const double* sA, const double* sB, int kg, int kn, int bstep,
                                        double (&acc)[8][4]) {
  switch (nu) {
    case 1: tn_stage<1, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
    case 2: tn_stage<2, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
    case 3: tn_stage<3, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
    case 4: tn_stage<4, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
    case 5: tn_stage<5, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
    case 6: tn_stage<6, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
    case 7: tn_stage<7, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
    default: tn_stage<8, NV, KG>(sA, sB, kg, kn, bstep, acc); break;
  }
}

template <int CG>
__global__ void __launch_bounds__(kThreads, 2)
k_gemm_tn(MatRef Y, MatRef C, int64_t m, int nb, int64_t n, int rt, int ct, int64_t kchunk, double* out,
          int64_t split_stride) {
  constexpr int KG = 8 / CG;
  __shared__ double sm[2 * 64 * kTnLd];
  double* sA = sm;                  // [column of Y][row], ld kTnLd
  double* sB = sm + 64 * kTnLd;     // [column of C][row]
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  // the two groups of CG = 4 pair column groups of different width on a sub-partition
  const int kg = warp / CG, g = (warp + 2 * kg) % CG;
  const int i0 = (int)blockIdx.x * rt;
  const int64_t j0 = (int64_t)blockIdx.y * ct;
  const int ni = nb - i0 < rt ? nb - i0 : rt;
  const int nj = (int)(n - j0 < ct ? n - j0 : ct);
  const int nu = (ni + 7) >> 3;
  const int nv = ((nj + 3) / 4 - g + CG - 1) / CG;   // column blocks of this warp
  const int64_t k0 = (int64_t)blockIdx.z * kchunk;
  const int64_t k1 = (k0 + kchunk < m) ? k0 + kchunk : m;
  double acc[8][4];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0.0;
  // element e of a stage: row kb + e % 32 of column e / 32; eight per thread and operand
  double pa[8], pb[8];
  const int kr = tid & 31, c0 = tid >> 5;
  const View vy = make_view(Y), vc = make_view(C);
  auto fetch = [&](int64_t kb) {
    const bool row = kb + kr < k1;
#pragma unroll
    for (int u = 0; u < 8; ++u) pa[u] = view_at(vy, kb + kr, i0 + c0 + 8 * u, row && c0 + 8 * u < ni);
#pragma unroll
    for (int u = 0; u < 2 * CG; ++u) pb[u] = view_at(vc, kb + kr, j0 + c0 + 8 * u, row && c0 + 8 * u < nj);
  };
  fetch(k0);
  const double* wa = sA + (lane & 7) * kTnLd;
  const double* wb = sB + (4 * g + (lane >> 3)) * kTnLd;
  constexpr int bstep = 4 * CG * kTnLd;
  for (int64_t kb = k0; kb < k1; kb += kTnK) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 8; ++u) sA[(c0 + 8 * u) * kTnLd + kr] = pa[u];
#pragma unroll
    for (int u = 0; u < 2 * CG; ++u) sB[(c0 + 8 * u) * kTnLd + kr] = pb[u];
    __syncthreads();
    if (kb + kTnK < k1) fetch(kb + kTnK);
    const int kn = (int)(k1 - kb < kTnK ? k1 - kb : kTnK);
    switch (nv) {
      case 4: tn_rows<4, KG>(nu, wa, wb, kg, kn, bstep, acc); break;
      case 3: tn_rows<3, KG>(nu, wa, wb, kg, kn, bstep, acc); break;
      case 2: tn_rows<2, KG>(nu, wa, wb, kg, kn, bstep, acc); break;
      case 1: tn_rows<1, KG>(nu, wa, wb, kg, kn, bstep, acc); break;
      default: break;
    }
  }
  // the groups' sums: the upper half of the groups hands its to the lower half
  constexpr int slot = 64 * 16 * CG;
#pragma unroll
  for (int h = KG / 2; h >= 1; h >>= 1) {
    __syncthreads();
    if (kg >= h && kg < 2 * h) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (u < nu) sm[(kg - h) * slot + ((u * 4 + v) * CG + g) * 32 + lane] = acc[u][v];
    }
    __syncthreads();
    if (kg < h) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (u >= nu) break;
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] += sm[kg * slot + ((u * 4 + v) * CG + g) * 32 + lane];
      }
    }
  }
  if (kg == 0) {
    double* o = out + (int64_t)blockIdx.z * split_stride;
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int i = 8 * u + (lane & 7), j = 4 * (v * CG + g) + (lane >> 3);
        if (i < ni && j < nj) o[(j0 + j) * nb + i0 + i] = acc[u][v];
      }
  }
}

// ---- C -= Y Z
//
// C (m x n, ldc) -= opY (m x nb) Z (nb x n, ldz): one row per lane, NC columns
// in registers, Z broadcast from shared memory (64 rows of it at a time) and Y
// read straight from memory, coalesced over the lanes, a few columns ahead.
// Rows and columns pad to 32 and 4.
constexpr int kNnK = 64;
constexpr int kNnThreads = 128;   // one warp per sub-partition: small products spread over the SMs

// One row's share of a stage for the first 4 NQ of NC columns; y holds the first
// PF columns of Y.
template <int NC, int NQ, int PF>
__device__ __forceinline__ void nn_stage(const View& vy, int64_t r, bool in, int kb, int kn, const double (*sZ)[NC],
                                         double (&y)[PF], double (&acc)[NC]) {
#pragma unroll 1
  for (int k = 0; k < kn; k += PF) {   // rows of sZ beyond kn are zero
    double x[PF];
#pragma unroll
    for (int u = 0; u < PF; ++u) x[u] = y[u];
#pragma unroll
    for (int u = 0; u < PF; ++u) y[u] = view_at(vy, r, kb + k + PF + u, in && k + PF + u < kn);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
#pragma unroll
      for (int u = 0; u < PF; ++u) {
        const double2 z0 = *reinterpret_cast<const double2*>(&sZ[k + u][4 * q]);
        const double2 z1 = *reinterpret_cast<const double2*>(&sZ[k + u][4 * q + 2]);
        acc[4 * q] = fma(x[u], z0.x, acc[4 * q]);
        acc[4 * q + 1] = fma(x[u], z0.y, acc[4 * q + 1]);
        acc[4 * q + 2] = fma(x[u], z1.x, acc[4 * q + 2]);
        acc[4 * q + 3] = fma(x[u], z1.y, acc[4 * q + 3]);
      }
    }
  }
}

template <int NC>
__global__ void __launch_bounds__(kNnThreads)
k_gemm_nn_sub(double* C, int64_t ldc, MatRef Y, MatRef Z, int64_t m, int64_t n, int nb) {
  constexpr int PF = NC >= 16 ? 4 : 8;             // columns of Y in flight: about 1000 cycles of FP64 work
  constexpr int per = kNnK * NC / kNnThreads;      // elements of a stage of Z per thread
  constexpr bool early = NC <= 16;                 // C's elements load before the products
  __shared__ __align__(16) double sZ[kNnK][NC];
  const int64_t r = (int64_t)blockIdx.x * kNnThreads + threadIdx.x;
  const int64_t j0 = (int64_t)blockIdx.y * NC;
  const int nj = (int)(n - j0 < NC ? n - j0 : NC);
  const bool in = r < m;
  const View vy = make_view(Y);
  double* c = C + j0 * ldc + r;
  double acc[NC], old[early ? NC : 1];
#pragma unroll
  for (int v = 0; v < NC; ++v) {
    acc[v] = 0.0;
    if constexpr (early) old[v] = (in && v < nj) ? c[v * ldc] : 0.0;
  }
  for (int kb = 0; kb < nb; kb += kNnK) {
    const int kn = nb - kb < kNnK ? nb - kb : kNnK;
    double y[PF], z[per];
#pragma unroll
    for (int u = 0; u < per; ++u) {
      const int e = threadIdx.x + kNnThreads * u, k = e % kNnK, j = e / kNnK;
      z[u] = (k < kn && j < nj) ? Z.p[(j0 + j) * Z.ld + kb + k] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < PF; ++u) y[u] = view_at(vy, r, kb + u, in && u < kn);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < per; ++u) {
      const int e = threadIdx.x + kNnThreads * u;
      sZ[e % kNnK][e / kNnK] = z[u];
    }
    __syncthreads();
    constexpr int Q = NC / 4;
    switch ((nj + 3) >> 2) {
      case 1: nn_stage<NC, 1, PF>(vy, r, in, kb, kn, sZ, y, acc); break;
      case 2: nn_stage<NC, (Q < 2 ? Q : 2), PF>(vy, r, in, kb, kn, sZ, y, acc); break;
      case 3: nn_stage<NC, (Q < 3 ? Q : 3), PF>(vy, r, in, kb, kn, sZ, y, acc); break;
      case 4: nn_stage<NC, (Q < 4 ? Q : 4), PF>(vy, r, in, kb, kn, sZ, y, acc); break;
      case 5: nn_stage<NC, (Q < 5 ? Q : 5), PF>(vy, r, in, kb, kn, sZ, y, acc); break;
      case 6: nn_stage<NC, (Q < 6 ? Q : 6), PF>(vy, r, in, kb, kn, sZ, y, acc); break;
      case 7: nn_stage<NC, (Q < 7 ? Q : 7), PF>(vy, r, in, kb, kn, sZ, y, acc); break;
      default: nn_stage<NC, Q, PF>(vy, r, in, kb, kn, sZ, y, acc); break;
    }
  }
  if (in) {
    if constexpr (early) {
#pragma unroll
      for (int v = 0; v < NC; ++v)
        if (v < nj) c[v * ldc] = old[v] - acc[v];
    } else {
#pragma unroll
      for (int v0 = 0; v0 < NC; v0 += 8) {
        if (v0 >= nj) break;
        double t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) t[u] = v0 + u < nj ? c[(v0 + u) * ldc] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (v0 + u < nj) c[(v0 + u) * ldc] = t[u] - acc[v0 + u];
      }
    }
  }
}

// Single-column forms (one right-hand side: Q^T b, Q b).  A 16 x 16 tile for
// one column would spend 15 of every 16 DFMAs on padding, so these run one
// FMA per element of Y, which is what bounds a matrix-vector product on the
// FP64 pipe.
//
// part[z * nb + i] = sum over the rows r of chunk z of Y(r, i) * c(r): one warp
// per column i of Y (lanes stride the rows, four accumulators), warp-reduced.
__global__ void __launch_bounds__(kThreads)
k_gemv_tn(MatRef Y, MatRef C, int64_t m, int nb, int64_t kchunk, double* part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * (kThreads / 32) + warp;
  if (i >= nb) return;   // warp-uniform
  const int64_t k0 = (int64_t)blockIdx.y * kchunk;
  const int64_t k1 = (k0 + kchunk < m) ? k0 + kchunk : m;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  int64_t r = k0 + lane;
  for (; r + 96 < k1; r += 128) {
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = fma(mat_at(Y, r + 32 * u, i), mat_at(C, r + 32 * u, 0), acc[u]);
  }
  for (; r < k1; r += 32) acc[0] = fma(mat_at(Y, r, i), mat_at(C, r, 0), acc[0]);
  const double sum = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
  if (lane == 0) part[(int64_t)blockIdx.y * nb + i] = sum;
}

// c(r) -= sum_k Y(r, k) z(k), one thread per row r (z staged in shared memory)
__global__ void __launch_bounds__(kThreads)
k_gemv_nn_sub(double* C, MatRef Y, const double* Z, int64_t m, int nb) {
  __shared__ double sz[256];
  for (int k = threadIdx.x; k < nb; k += kThreads) sz[k] = Z[k];
  __syncthreads();
  const int64_t r = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (r >= m) return;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  int k = 0;
  for (; k + 4 <= nb; k += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = fma(mat_at(Y, r, k + u), sz[k + u], acc[u]);
  }
  for (; k < nb; ++k) acc[0] = fma(mat_at(Y, r, k), sz[k], acc[0]);
  C[r] -= (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

// Small-matrix product, 16 x 16 outputs per CTA, one per thread:
// C(i,j) = alpha * sum_k opA(i,k) opB(k,j) + beta * C(i,j)   (beta == 0: C not read).
__global__ void __launch_bounds__(kThreads)
k_small_gemm(MatRef A, MatRef B, int64_t M, int64_t N, int64_t K, double alpha, double beta,
             double* C, int64_t ldc) {
  __shared__ double sA[16][65];
  __shared__ double sB[64][17];
  const int ti = threadIdx.x % 16, tj = threadIdx.x / 16;
  const int64_t i0 = (int64_t)blockIdx.x * 16, j0 = (int64_t)blockIdx.y * 16;
  double acc = 0.0;
  for (int64_t kb = 0; kb < K; kb += 64) {
    for (int idx = threadIdx.x; idx < 16 * 64; idx += kThreads) {
      int ii = idx % 16, kk = idx / 16;
      int64_t gi = i0 + ii, gk = kb + kk;
      sA[ii][kk] = (gi < M && gk < K) ? mat_at(A, gi, gk) : 0.0;
      int jj = idx / 64, k2 = idx % 64;
      int64_t gj = j0 + jj, gk2 = kb + k2;
      sB[k2][jj] = (gj < N && gk2 < K) ? mat_at(B, gk2, gj) : 0.0;
    }
    __syncthreads();
    const int kn = (int)(K - kb < 64 ? K - kb : 64);
    for (int k0 = 0; k0 < kn; k0 += 8) {   // zeros beyond K
#pragma unroll
      for (int kk = k0; kk < k0 + 8; ++kk) acc = fma(sA[ti][kk], sB[kk][tj], acc);
    }
    __syncthreads();
  }
  int64_t gi = i0 + ti, gj = j0 + tj;
  if (gi < M && gj < N) {
    double v = alpha * acc;
    if (beta != 0.0) v += beta * C[gj * ldc + gi];
    C[gj * ldc + gi] = v;
  }
}

// T12 = -T11 G T22 of two upper-triangular factors (T11: b1 x b1, T22: b2 x b2, T12
// beside them with the same ld) and G (b1 x b2, ld b1).  One CTA per column j, as
// in k_reduce_apply: thread (i, g) takes every 256 / nbp-th term of row i, first of
// t = G T22(:, j), then of T11 t.  One launch of 6 us where two small products took
// 9 each (bound by the latencies of loads and of the FP64 pipe).
__global__ void __launch_bounds__(kThreads)
k_merge_t(const double* G, double* T, int64_t ldT, int b1, int b2, int nbp) {
  __shared__ double part[kThreads];
  __shared__ double col[kThreads];
  const int NG = kThreads / nbp;
  const int i = threadIdx.x % nbp, g = threadIdx.x / nbp, j = blockIdx.x;
  const double* t22 = T + (int64_t)(b1 + j) * ldT + b1;
  double v = 0.0;
  for (int k0 = 0; k0 <= j; k0 += kThreads) {   // b2 may exceed kThreads (an odd width's wider half)
    const int kn = j + 1 - k0 < kThreads ? j + 1 - k0 : kThreads;
    if (k0) __syncthreads();
    if ((int)threadIdx.x < kn) col[threadIdx.x] = t22[k0 + threadIdx.x];
    __syncthreads();
    if (i < b1)
      for (int k = g; k < kn; k += NG) v = fma(G[(int64_t)(k0 + k) * b1 + i], col[k], v);
  }
  part[g * nbp + i] = v;
  __syncthreads();
  if (g == 0) {
    double t = 0.0;
    for (int h = 0; h < NG; ++h) t += part[h * nbp + i];
    col[i] = t;
  }
  __syncthreads();
  v = 0.0;
  for (int k = i + g; k < b1; k += NG) v = fma(T[(int64_t)k * ldT + i], col[k], v);
  part[g * nbp + i] = v;
  __syncthreads();
  if (g == 0 && i < b1) {
    double t = 0.0;
    for (int h = 0; h < NG; ++h) t += part[h * nbp + i];
    T[(int64_t)(b1 + j) * ldT + i] = -t;
  }
}

// Z(i,j) = alpha * sum_k opT(i,k) * (sum_s Zp[s](k,j))   with Zp[s] nb x n (ld nb);
// opT == nullptr: identity.  One CTA per output column j; thread (i, g) of the
// (nbp rows) x (256 / nbp groups) layout sums every G-th partial of row i, the
// groups are combined in shared memory, and the product with opT splits its k
// range over the groups the same way, so every dependent FP64 chain is about
// nsplit / G + nb / G long instead of nsplit + nb.  The summation order is
// fixed, so the result is deterministic.  With few columns of 128 rows or more a CTA
// has 1024 threads: its loads and FP64 chains bound the launch then (a 128 x 16
// step of a triangular solve with 32 partials: 17 + 6 us as a product and a
// reduction, 8 here).
template <int TH>
__global__ void __launch_bounds__(TH)
k_reduce_apply(const double* Zp, int nsplit, int64_t split_stride, int nb, int nbp, int64_t n,
               MatRef Top, double alpha, double* Z, int64_t ldz) {
  __shared__ double part[TH];
  __shared__ double col[256];
  const int G = TH / nbp;
  const int i = threadIdx.x % nbp, g = threadIdx.x / nbp;
  const int64_t jc = blockIdx.x;
  double sacc = 0.0;
  if (i < nb)
    for (int sp = g; sp < nsplit; sp += G) sacc += Zp[sp * split_stride + jc * nb + i];
  part[g * nbp + i] = sacc;
  __syncthreads();
  if (g == 0) {
    double t = 0.0;
    for (int h = 0; h < G; ++h) t += part[h * nbp + i];
    col[i] = t;
  }
  __syncthreads();
  double z;
  if (Top.p == nullptr) {
    z = (g == 0 && i < nb) ? col[i] : 0.0;
  } else {
    z = 0.0;
    if (i < nb)
      for (int k = g; k < nb; k += G) z = fma(mat_at(Top, i, k), col[k], z);
  }
  __syncthreads();
  part[g * nbp + i] = z;
  __syncthreads();
  if (g == 0 && i < nb) {
    double t = 0.0;
    for (int h = 0; h < G; ++h) t += part[h * nbp + i];
    Z[jc * ldz + i] = alpha * t;
  }
}

// Triangular inverses: batch q inverts the n_q x n_q triangle at X + q xstep,
// n_q = min(n, ntot - q n), into the n x n block Xi + q istep (zero outside the
// triangle).  lower != 0: lower triangular, worked as the transpose of an upper
// one; unit != 0: unit diagonal implied.
// One warp per column of the inverse (four a CTA), blocked back substitution
// with one row per lane: the CTA stages 32 x 32 blocks of the triangle (the
// next one loads while this one is used), a block above the diagonal costs 32
// FP64 instructions a column and a diagonal block, its columns divided by the
// diagonal first, a chain of 32 shuffles and fmas.  Bound by those chains: 28 us
// at n = 128, where a thread per column took 480 us (600 us for the diagonal
// blocks of a least-squares R).
// Element (i, c) of the inverse depends on rows and columns i..c only, but the blocks
// multiply by whole columns and by reciprocals: a column that comes out non-finite, or
// that used a pivot outside 2^+-200 (where a quotient could leave the normal range), is
// worked again by itself (tri_column).
constexpr int kTriWarps = 4;

// Column c of the inverse of the upper triangle X(i, k) = X[i xi + k xk] into x[i xs],
// i <= c: plain back substitution by one warp, every entry divided where it is used.
__device__ __noinline__ void tri_column(const double* X, int64_t xi, int64_t xk, int unit, int c, double* x, int64_t xs) {
  const int lane = threadIdx.x & 31;
  for (int i = lane; i <= c; i += 32) x[i * xs] = i == c ? 1.0 : 0.0;
  for (int k = c; k >= 0; --k) {
    __syncwarp();
    double v = x[k * xs];
    if (!unit) v /= X[k * (xi + xk)];
    __syncwarp();
    if (lane == 0) x[k * xs] = v;
    for (int i = lane; i < k; i += 32) x[i * xs] = fma(-X[i * xi + k * xk], v, x[i * xs]);
  }
}

__global__ void __launch_bounds__(32 * kTriWarps)
k_tri_inv(const double* X, int64_t ldx, int n, int64_t ntot, int64_t xstep, int lower, int unit, double* Xi,
          int64_t ldi, int64_t istep) {
  constexpr int ld = 33, per = 1024 / (32 * kTriWarps);
  __shared__ double sU[32 * ld];
  __shared__ double s_rd[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t q = blockIdx.y;
  X += q * xstep;
  Xi += q * istep;
  const int nq = (int)(ntot - q * n < n ? ntot - q * n : n);
  const int c = blockIdx.x * kTriWarps + warp, J = blockIdx.x * kTriWarps / 32;
  const int64_t ri = lower ? ldi : 1, ci = lower ? 1 : ldi;     // strides of the upper view of Xi
  // element (i, k) of the upper view of block (ib, kb); identity beyond nq
  auto at = [&](int ib, int kb, int e) -> double {
    const int i = 32 * ib + (lower ? e >> 5 : e & 31), k = 32 * kb + (lower ? e & 31 : e >> 5);
    if (i < k && k < nq) return lower ? X[i * ldx + k] : X[k * ldx + i];
    if (i == k) return (i < nq && !unit) ? X[i * ldx + i] : 1.0;
    return 0.0;
  };
  double nxt[per];
  auto fetch = [&](int ib, int kb) {
#pragma unroll
    for (int u = 0; u < per; ++u) nxt[u] = at(ib, kb, tid + 32 * kTriWarps * u);
  };
  auto stage = [&]() {
#pragma unroll
    for (int u = 0; u < per; ++u) {
      const int e = tid + 32 * kTriWarps * u;
      sU[lower ? (e & 31) * ld + (e >> 5) : (e >> 5) * ld + (e & 31)] = nxt[u];
    }
  };
  if (c < n)
    for (int i = 32 * (J + 1) + lane; i < n; i += 32) Xi[i * ri + c * ci] = 0.0;
  bool again = false;   // this lane's entries, or pivots of the blocks passed
  fetch(J, J);
  for (int ib = J; ib >= 0; --ib) {
    const int i = 32 * ib + lane;
    double r0 = (i == c && c < nq) ? 1.0 : 0.0, r1 = 0.0;
    for (int kb = J; kb > ib; --kb) {
      __syncthreads();
      stage();
      if (kb - 1 >= ib) fetch(ib, kb - 1);
      __syncthreads();
      const int kk = 32 * kb + lane;
      const double x = (c < n && kk < n) ? Xi[kk * ri + c * ci] : 0.0;
#pragma unroll 8
      for (int k = 0; k < 32; k += 2) {
        r0 = fma(-sU[k * ld + lane], __shfl_sync(0xffffffffu, x, k), r0);
        r1 = fma(-sU[(k + 1) * ld + lane], __shfl_sync(0xffffffffu, x, k + 1), r1);
      }
    }
    __syncthreads();
    stage();
    if (ib > 0) fetch(ib - 1, J);
    __syncthreads();
    if (tid < 32) s_rd[tid] = 1.0 / sU[tid * ld + tid];
    __syncthreads();
    // columns k divided by U[k][k]: r_i -= (U[i][k] / U[k][k]) r_k, then x = r / diag
#pragma unroll
    for (int u = 0; u < per; ++u) {
      const int e = tid + 32 * kTriWarps * u, k = e >> 5;
      sU[k * ld + (e & 31)] *= s_rd[k];
    }
    __syncthreads();
    double r = r0 + r1;
#pragma unroll 8
    for (int k = 31; k > 0; --k) {
      const double rk = __shfl_sync(0xffffffffu, r, k);
      if (lane < k) r = fma(-sU[k * ld + lane], rk, r);
    }
    const double rd = s_rd[lane], x = r * rd;
    again |= ((unsigned)__double2hiint(x) & 0x7fffffffu) >= 0x7ff00000u ||
             ((unsigned)__double2hiint(rd) & 0x7fffffffu) - ((1023u - 200u) << 20) > (400u << 20);
    if (c < n && i < n) Xi[i * ri + c * ci] = x;
    __syncwarp();
  }
  if (!__any_sync(0xffffffffu, again) || c >= nq) return;
  for (int i = c + 1 + lane; i < 32 * (J + 1) && i < n; i += 32) Xi[i * ri + c * ci] = 0.0;
  tri_column(X, lower ? ldx : 1, lower ? 1 : ldx, unit, c, Xi + c * ci, ri);
}

// Copy op(X) (masked) into a dense n x k buffer (ld ldo).
__global__ void k_materialize(MatRef X, int64_t n, int64_t k, double* out, int64_t ldo) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n * k) return;
  int64_t i = idx % n, j = idx / n;
  out[j * ldo + i] = mat_at(X, i, j);
}

// T^-T from a Gram matrix: lower part of G with halved diagonal (qr_2d.cxx:46-51);
// only the lower triangle (incl. diagonal) of T is written, as unpack_lower does.
__global__ void k_invT_from_gram(const double* G, int64_t ldg, int b, double* T, int64_t ldt) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= b * b) return;
  int i = idx % b, j = idx / b;
  if (i < j) return;
  double g = G[(int64_t)j * ldg + i];
  T[(int64_t)j * ldt + i] = (i == j) ? 0.5 * g : g;
}

// out (n x k, ld) = identity (ones on the leading diagonal, zeros elsewhere)
__global__ void k_set_identity(double* out, int64_t ld, int64_t n, int64_t k) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n * k) return;
  int64_t i = idx % n, j = idx / n;
  out[j * ld + i] = (i == j) ? 1.0 : 0.0;
}

// ---------------------------------------------------------------- host side

static int num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

int small_gemm(int64_t M, int64_t N, int64_t K, double alpha, MatRef A, MatRef B, double beta,
               double* C, int64_t ldc, cudaStream_t s) {
  if (M <= 0 || N <= 0) return CANDMC_OK;
  dim3 grid((unsigned)((M + 15) / 16), (unsigned)((N + 15) / 16));
  ProfScope ps(CANDMC_KCLASS_SMALL, 2.0 * M * N * K, s);
  k_small_gemm<<<grid, kThreads, 0, s>>>(A, B, M, N, K, alpha, beta, C, ldc);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

int merge_t(const double* G, double* T, int64_t ldT, int b1, int b2, cudaStream_t s) {
  if (b1 > kThreads) return set_error(CANDMC_ERR_ARG, "merge_t needs a first factor of at most 256 columns");
  int nbp = 1;
  while (nbp < b1) nbp <<= 1;
  ProfScope ps(CANDMC_KCLASS_SMALL, 2.0 * b1 * b2 * (b1 + b2), s);
  k_merge_t<<<(unsigned)b2, kThreads, 0, s>>>(G, T, ldT, b1, b2, nbp);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

// Z = alpha opT (sum of the nsplit partial products)
int reduce_apply(const double* part, int64_t nsplit, int64_t stride, int nb, int64_t n, MatRef Top,
                        double alpha, double* Z, int64_t ldz, cudaStream_t s) {
  int nbp = 1;
  while (nbp < nb) nbp <<= 1;
  ProfScope ps(CANDMC_KCLASS_REDUCE, 8.0 * stride * nsplit, s);
  if (nbp >= 128 && n <= 2 * num_sms())
    k_reduce_apply<1024><<<(unsigned)n, 1024, 0, s>>>(part, (int)nsplit, stride, nb, nbp, n, Top, alpha, Z, ldz);
  else
    k_reduce_apply<kThreads><<<(unsigned)n, kThreads, 0, s>>>(part, (int)nsplit, stride, nb, nbp, n, Top, alpha, Z, ldz);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

static int small_tn(MatRef Y, MatRef C, int64_t m, int nb, int64_t n, MatRef Top, double alpha, double* Z,
                    int64_t ldz, cudaStream_t s) {
  // about 4 CTAs per SM over slices of TK rows or more
  const int64_t tiles = (int64_t)((nb + 15) / 16) * ((n + 15) / 16), target = 4 * (int64_t)num_sms();
  int64_t nsplit = std::max<int64_t>(1, std::min<int64_t>((target + tiles - 1) / tiles, (m + TK - 1) / TK));
  const int64_t kchunk = ((m + nsplit - 1) / nsplit + TK - 1) / TK * TK;
  nsplit = std::max<int64_t>(1, (m + kchunk - 1) / kchunk);
  const int64_t stride = (int64_t)nb * n;
  DevBuf part;
  CANDMC_RET(part.alloc(sizeof(double) * (size_t)stride * nsplit, s));
  MatRef Yt = Y;
  Yt.trans = !Y.trans;   // element (i, r) of Y^T is Y(r, i)
  {
    ProfScope ps(CANDMC_KCLASS_GEMM_TN, 2.0 * nb * n * m, s);
    const dim3 grid((unsigned)((nb + 15) / 16), (unsigned)((n + 15) / 16), (unsigned)nsplit);
    k_gemm_f64<<<grid, kThreads, 0, s>>>(Yt, C, nb, n, m, kchunk, part.d(), nb, stride, 0);
  }
  CANDMC_CK(cudaGetLastError());
  return reduce_apply(part.d(), nsplit, stride, nb, n, Top, alpha, Z, ldz, s);
}

// Z (nb x n, ldz) = alpha * opT * (opY^T * opC), Y and C with m rows.
// opT.p == nullptr means no triangular factor.
int gemm_tn_reduce(MatRef Y, MatRef C, int64_t m, int nb, int64_t n, MatRef Top, double alpha,
                   double* Z, int64_t ldz, cudaStream_t s) {
  if (nb <= 0 || n <= 0) return CANDMC_OK;
  if (nb > 256) return CANDMC_ERR_ARG;
  if (n == 1) {
    // one column: a warp per column of Y over row slices, about 8 CTAs per SM
    const int64_t cblk = (nb + kThreads / 32 - 1) / (kThreads / 32);
    int64_t nsplit = std::max<int64_t>(1, std::min<int64_t>((8 * (int64_t)num_sms() + cblk - 1) / cblk,
                                                            (m + 255) / 256));
    int64_t kchunk = (m + nsplit - 1) / nsplit;
    nsplit = std::max<int64_t>(1, (m + kchunk - 1) / kchunk);
    DevBuf part;
    CANDMC_RET(part.alloc(sizeof(double) * (size_t)nb * nsplit, s));
    {
      ProfScope ps(CANDMC_KCLASS_GEMM_TN, 2.0 * nb * m, s);
      k_gemv_tn<<<dim3((unsigned)cblk, (unsigned)nsplit), kThreads, 0, s>>>(Y, C, m, nb, kchunk, part.d());
    }
    CANDMC_CK(cudaGetLastError());
    return reduce_apply(part.d(), nsplit, nb, nb, 1, Top, alpha, Z, ldz, s);
  }
  // (small_tn's grid takes 65535 tiles of 16 columns; the product below goes in pieces)
  if (m * nb * n <= kSmallProduct && n <= 16 * (int64_t)65535) return small_tn(Y, C, m, nb, n, Top, alpha, Z, ldz, s);
  // column groups: 4, or 1 (and eight groups of rows) when there are at most
  // two column blocks; row tiles of at most 64 rows, all alike
  const int cg = n > 8 ? 4 : 1;
  int ntr = (nb + 63) / 64, rt = ((nb + ntr - 1) / ntr + 7) / 8 * 8, ct = 16 * cg;
  auto ntiles = [&]() { return (int64_t)((nb + rt - 1) / rt) * ((n + ct - 1) / ct); };
  // FP64 work per CTA is what bounds these kernels: full waves of 2 CTAs per
  // SM, or 1 when their chunks would be shorter than 128 rows.  Chunks shorter
  // than 64 rows take smaller tiles instead, which leaves fewer partial sums to
  // add (2000 x 64 x 64: 16 x 32 tiles and 19 chunks, not 125).
  const int64_t sms = num_sms(), target = sms * (m * ntiles() >= 256 * sms ? 2 : 1);
  while (m * ntiles() < 64 * sms && (rt > 16 || ct > 16)) {
    if (rt >= ct && rt > 16) rt = (rt / 2 + 7) / 8 * 8;
    else if (ct > 16) ct /= 2;
    else break;
  }
  const int64_t tiles = ntiles();
  int64_t nsplit = std::max<int64_t>(1, std::min<int64_t>(target / tiles, (m + 15) / 16));
  nsplit = std::min<int64_t>(nsplit, 1024);
  if (nsplit <= 4) {
    // Many tiles: CTAs on one SM share its FP64 pipe, so the fullest SM's rows
    // count, and a split that leaves it few more than the mean is worth its
    // partials (a CTA's start and end cost about 24 rows, adding a partial 4).
    // 2048 x 128 x 16384, 512 tiles: one chunk 8.45 ms (4 rounds where 3.37 would
    // do), 2 chunks 7.35; 16384 x 128 x 8192, 256 tiles: 34.3, and 28.7 with 7.
    int64_t best = INT64_MAX;
    for (int64_t ns = 1; ns <= 8 && (ns == 1 || m / ns >= 128); ++ns) {
      const int64_t cost = (tiles * ns + sms - 1) / sms * ((m + ns - 1) / ns + 24) + 4 * ns;
      if (cost < best) {
        best = cost;
        nsplit = ns;
      }
    }
  }
  const int64_t kchunk = (m + nsplit - 1) / nsplit;
  nsplit = std::max<int64_t>(1, (m + kchunk - 1) / kchunk);
  const int64_t stride = (int64_t)nb * n;
  DevBuf part;
  CANDMC_RET(part.alloc(sizeof(double) * (size_t)stride * nsplit, s));
  {
    ProfScope ps(CANDMC_KCLASS_GEMM_TN, 2.0 * nb * n * m, s);
    // grid rows are limited to 65535 column tiles a launch
    for (int64_t jt = 0; jt < n; jt += 65535 * (int64_t)ct) {
      const int64_t nn = std::min<int64_t>(n - jt, 65535 * (int64_t)ct);
      MatRef Cj = C;
      Cj.p = C.p + (C.trans ? jt : jt * C.ld);
      Cj.off = C.trans ? C.off - jt : C.off + jt;
      const dim3 grid((unsigned)((nb + rt - 1) / rt), (unsigned)((nn + ct - 1) / ct), (unsigned)nsplit);
      double* o = part.d() + jt * nb;
      if (cg == 4) k_gemm_tn<4><<<grid, kThreads, 0, s>>>(Y, Cj, m, nb, nn, rt, ct, kchunk, o, stride);
      else k_gemm_tn<1><<<grid, kThreads, 0, s>>>(Y, Cj, m, nb, nn, rt, ct, kchunk, o, stride);
    }
  }
  CANDMC_CK(cudaGetLastError());
  return reduce_apply(part.d(), nsplit, stride, nb, n, Top, alpha, Z, ldz, s);
}

// C (m x n, ldc) -= opY (m x nb) * Z (nb x n, ldz)
int gemm_nn_sub(double* C, int64_t ldc, MatRef Y, const double* Z, int64_t ldz, int64_t m, int64_t n,
                int nb, cudaStream_t s) {
  if (m <= 0 || n <= 0 || nb <= 0) return CANDMC_OK;
  if (n == 1 && nb <= 256) {
    ProfScope ps(CANDMC_KCLASS_GEMM_NN, 2.0 * m * nb, s);
    k_gemv_nn_sub<<<(unsigned)((m + kThreads - 1) / kThreads), kThreads, 0, s>>>(C, Y, Z, m, nb);
    CANDMC_CK(cudaGetLastError());
    return CANDMC_OK;
  }
  if (m * n * nb <= kSmallProduct && n <= 16 * (int64_t)65535) {
    ProfScope ps(CANDMC_KCLASS_GEMM_NN, 2.0 * m * n * nb, s);
    const dim3 grid((unsigned)((m + 15) / 16), (unsigned)((n + 15) / 16));
    k_gemm_f64<<<grid, kThreads, 0, s>>>(Y, mref(Z, ldz), m, n, nb, nb, C, ldc, 0, 1);
    CANDMC_CK(cudaGetLastError());
    return CANDMC_OK;
  }
  // columns per CTA: the fewest column times on the fullest SM (a CTA is one
  // warp per sub-partition)
  const int64_t rb = (m + kNnThreads - 1) / kNnThreads, sms = num_sms();
  auto cost = [&](int64_t nc) { return (rb * ((n + nc - 1) / nc) + sms - 1) / sms * std::min<int64_t>(nc, (n + 3) / 4 * 4); };
  int nc = 32;
  for (int t : {16, 8, 4})
    if (cost(t) < cost(nc)) nc = t;
  ProfScope ps(CANDMC_KCLASS_GEMM_NN, 2.0 * m * n * nb, s);
  // grid columns are limited to 65535
  for (int64_t j = 0; j < n; j += 65535 * (int64_t)nc) {
    const int64_t nn = std::min<int64_t>(n - j, 65535 * (int64_t)nc);
    const dim3 grid((unsigned)rb, (unsigned)((nn + nc - 1) / nc));
    const MatRef Zm = mref(Z + j * ldz, ldz);
    if (nc == 32) k_gemm_nn_sub<32><<<grid, kNnThreads, 0, s>>>(C + j * ldc, ldc, Y, Zm, m, nn, nb);
    else if (nc == 16) k_gemm_nn_sub<16><<<grid, kNnThreads, 0, s>>>(C + j * ldc, ldc, Y, Zm, m, nn, nb);
    else if (nc == 8) k_gemm_nn_sub<8><<<grid, kNnThreads, 0, s>>>(C + j * ldc, ldc, Y, Zm, m, nn, nb);
    else k_gemm_nn_sub<4><<<grid, kNnThreads, 0, s>>>(C + j * ldc, ldc, Y, Zm, m, nn, nb);
  }
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

int tri_inv(const double* X, int64_t ldx, int n, int lower, int unit, double* Xi, int64_t ldi,
            cudaStream_t s) {
  if (n <= 0) return CANDMC_OK;
  ProfScope ps(CANDMC_KCLASS_SMALL, 0.0, s);
  k_tri_inv<<<(n + kTriWarps - 1) / kTriWarps, 32 * kTriWarps, 0, s>>>(X, ldx, n, n, 0, lower, unit, Xi, ldi, 0);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

int diag_inv(const double* R, int64_t ldr, int64_t n, int w, double* Dinv, cudaStream_t s) {
  const int64_t nblk = (n + w - 1) / w;
  // grid rows are limited to 65535 blocks a launch
  for (int64_t q = 0; q < nblk; q += 65535) {
    const int64_t cnt = std::min<int64_t>(65535, nblk - q);
    ProfScope ps(CANDMC_KCLASS_SMALL, 0.0, s);
    k_tri_inv<<<dim3((w + kTriWarps - 1) / kTriWarps, (unsigned)cnt), 32 * kTriWarps, 0, s>>>(
        R + q * w * (ldr + 1), ldr, w, n - q * w, w * (ldr + 1), 0, 0, Dinv + q * (int64_t)w * w, w, (int64_t)w * w);
    CANDMC_CK(cudaGetLastError());
  }
  return CANDMC_OK;
}

int materialize(MatRef X, int64_t n, int64_t k, double* out, int64_t ldo, cudaStream_t s) {
  if (n <= 0 || k <= 0) return CANDMC_OK;
  int64_t tot = n * k;
  ProfScope ps(CANDMC_KCLASS_SMALL, 16.0 * tot, s);
  k_materialize<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(X, n, k, out, ldo);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

int set_identity(double* out, int64_t ld, int64_t n, int64_t k, cudaStream_t s) {
  if (n <= 0 || k <= 0) return CANDMC_OK;
  int64_t tot = n * k;
  ProfScope ps(CANDMC_KCLASS_SMALL, 8.0 * tot, s);
  k_set_identity<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(out, ld, n, k);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

int invT_from_gram(const double* G, int64_t ldg, int b, double* T, int64_t ldt, cudaStream_t s) {
  if (b <= 0) return CANDMC_OK;
  ProfScope ps(CANDMC_KCLASS_SMALL, 0.0, s);
  k_invT_from_gram<<<(b * b + 255) / 256, 256, 0, s>>>(G, ldg, b, T, ldt);
  CANDMC_CK(cudaGetLastError());
  return CANDMC_OK;
}

}  // namespace candmc
