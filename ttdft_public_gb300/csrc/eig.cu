// Largest r eigenpairs of a symmetric n x n matrix in FP64: the mode Gram
// matrices of the sequentially truncated HOSVD (TuckerMPI::STHOSVD as used
// at main.cc:951-955 and ProjectHamiltonianSparse.cc:1113-1118), whose
// eigenvalues span ~14 orders of magnitude, so that an FP32 eigensolver
// cannot resolve the truncation subspace.
//
// FP64 runs at a small fraction of the FP32 rate on this GPU, so no stage is
// left to a single SM:
//
//  1. Householder tridiagonalisation A = Q T Q^T by one cluster of CTAs
//     (k_tridiag_cluster): every CTA keeps its rows of A on the SM, one cluster
//     barrier per column.
//  2. Eigenvalues by multisection on Sturm counts: one CTA per eigenvalue,
//     128 points per round (bisection would take 52 rounds to reach FP64
//     resolution, multisection 8).
//  3. Eigenvectors of T by inverse iteration (tridiagonal LU with partial
//     pivoting, three passes; equal eigenvalues are separated by a small
//     shift perturbation as in LAPACK's dstein), then u = Q z by applying
//     the stored reflectors in reverse order: one warp per eigenvector.
//  4. Orthonormalisation.  The vectors are orthonormal to ~1e-8 or better
//     except within clusters of eigenvalues.  With S = U^T U = I + E and
//     max |E| <= 1e-8 one Newton-Schulz step U <- U (3 I - S) / 2 leaves an
//     error of E^2; otherwise U <- U L^-T with S = L L^T, twice (Cholesky
//     QR2), with a Gram-Schmidt fallback if a Cholesky pivot fails.

#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>

#include "ttg_internal.cuh"

namespace cg = cooperative_groups;

namespace ttg {
namespace {

constexpr int kTrThreads = 512;
constexpr int kTrWarps = kTrThreads / 32;
constexpr int kVecWarps = 4;              // warps of the vector stage: 128 threads
constexpr int kMaxCluster = 16;
constexpr int kMaxN = 2048;
constexpr size_t kTrMaxSmem = 226 * 1024;

__device__ double cta_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += red[i];
  return s;
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sum over the 128 threads of the vector stage (named barrier 1)
__device__ __forceinline__ double vec_sum(double v, double* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  asm volatile("bar.sync 1, %0;" ::"n"(kVecWarps * 32) : "memory");
  return (red[0] + red[1]) + (red[2] + red[3]);
}

// 1/sqrt(x) and 1/x in FP64: an FP32 start and one step of Householder's
// third-order method (relative error e^3 < 1e-17) for x well inside the FP32
// range, else the CUDA functions.  The FP64 pipe has two lanes per SM, so the
// serial chains below count its operations.
__device__ __forceinline__ double fast_rsqrt(double x) {
  const float f = (float)x;
  if (!(f > 1e-30f && f < 1e30f)) return 1.0 / sqrt(x);
  const double y = (double)rsqrtf(f);
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

__device__ __forceinline__ double fast_inv(double x) {
  const float f = (float)x, a = fabsf(f);
  if (!(a > 1e-30f && a < 1e30f)) return 1.0 / x;
  const double y = (double)(1.0f / f);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// x / y; a reciprocal of its own where y is well inside the FP32 range (beyond
// it 1 / y may overflow where x / y does not)
__device__ __forceinline__ double fast_div(double x, double y) {
  const float a = fabsf((float)y);
  return a > 1e-30f && a < 1e30f ? x * fast_inv(y) : x / y;
}

// Largest v over the 128 threads of the vector stage (named barrier 1).
__device__ __forceinline__ int vec_max(int v, double* red) {
  v = __reduce_max_sync(0xffffffffu, v);
  int* m = reinterpret_cast<int*>(red);
  if ((threadIdx.x & 31) == 0) m[threadIdx.x >> 5] = v;
  asm volatile("bar.sync 1, %0;" ::"n"(kVecWarps * 32) : "memory");
  return max(max(m[0], m[1]), max(m[2], m[3]));
}

// The column v[j + 1 .. n) scaled by a power of two to a largest entry near 1;
// its square, and the exponent taken out (0 for zeros and non-finite values).
// By the 128 threads of the vector stage; a rare path, kept out of the loop.
__device__ __noinline__ double scale_column(double* v, int j, int n, double ss, double (*red)[kVecWarps],
                                            int& ex) {
  int m = 0;                                        // largest biased exponent
  for (int r = j + 1 + threadIdx.x; r < n; r += kVecWarps * 32)
    m = max(m, (__double2hiint(v[r]) >> 20) & 0x7ff);
  m = vec_max(m, red[1]);
  if (m == 0 || m == 0x7ff) return ss;
  ex = m - 1023;
  ss = 0.0;
  for (int r = j + 1 + threadIdx.x; r < n; r += kVecWarps * 32) {
    const double x = ldexp(v[r], -ex);
    v[r] = x;
    ss = fma(x, x, ss);
  }
  return vec_sum(ss, red[0]);
}

// Stage 1.  A (n x n column-major, symmetric); outputs the diagonal d,
// off-diagonal e (e[i] couples i and i+1), tau and the reflectors Vr (column
// j holds v_j in rows j+1..n-1).
//
// Row r of A belongs to CTA r mod C of the cluster: in shared memory (SM; the
// whole cluster holds 16 x 226 KB), or for larger n in A itself (its column r,
// L2 and L1 of that SM).  Per column j:
//  - vector stage, redundantly on every CTA (four warps): the column x_j of
//    the updated matrix -> reflector v_j, tau_j.  A column whose square is far
//    from 1 is first scaled by a power of two, which the reflector does not see:
//    the columns of a matrix of low rank can fall by 1e-16 each, down to where
//    1 / |v|^2 overflows;
//  - pass over the CTA's rows, a warp per row: the rank-2 update of column
//    j - 1 (B -= v w^T + w v^T) and p = tau B v_j in one sweep, three FP64 FMAs
//    an element; each row's p_r and its entry of column j + 1 go to every CTA
//    (distributed shared memory, two buffers);
//  - one cluster barrier; then w = p - (tau/2)(v.p) v, and column j + 1 follows
//    from its entries before the update: x = c - v w_{j+1} - w v_{j+1}.
// Bound by the FP64 pipe of the cluster's SMs (n^3 FMAs) and about 1.6 us a
// column for the vector stage and the barrier.  Before, the rows stayed in L2,
// each column took two barriers, two sweeps and CTA-wide sums that cost 4 us.
// Measured: n = 360: 7.6 -> 2.36 ms; n = 160: 2.74 -> 0.65; n = 1,200 (rows in
// L2): 103 -> 40.
template <bool SM>
__global__ void __launch_bounds__(kTrThreads) k_tridiag_cluster(
    double* __restrict__ A, int n, double* __restrict__ d, double* __restrict__ e,
    double* __restrict__ tau, double* __restrict__ Vr) {
  cg::cluster_group cl = cg::this_cluster();
  const int q = (int)cl.block_rank(), C = (int)cl.num_blocks();
  extern __shared__ double sm[];
  double* V0 = sm;                                  // v_j and x_{j+1} by turns
  double* V1 = V0 + n;
  double* wp = V1 + n;                              // w of the column before
  double* pb = wp + n;                              // 2 x n: p of all rows
  double* cb = pb + 2 * n;                          // 2 x n: column j + 1 of all rows
  double* rows = cb + 2 * n;
  __shared__ double red[2][kVecWarps];
  __shared__ double s_tau;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nloc = (n - q + C - 1) / C;             // rows q, q + C, ...
  if constexpr (SM)
    for (int i = warp; i < nloc; i += kTrWarps)
      for (int c = lane; c < n; c += 32) rows[(int64_t)i * n + c] = A[(int64_t)(q + i * C) * n + c];
  for (int r = tid; r < n; r += kTrThreads) {
    V0[r] = A[r];                                   // column 0
    V1[r] = 0.0;
    wp[r] = 0.0;
  }
  if (q == 0 && tid == 0) d[0] = A[0];
  __syncthreads();
  cl.sync();                                        // every CTA runs before remote writes
  for (int j = 0; j + 2 < n; ++j) {
    double* v = (j & 1) ? V1 : V0;                  // x_j on entry
    double* vprev = (j & 1) ? V0 : V1;
    if (warp < kVecWarps) {
      double ss = 0.0;
      for (int r = j + 1 + tid; r < n; r += kVecWarps * 32) ss = fma(v[r], v[r], ss);
      ss = vec_sum(ss, red[0]);
      int ex = 0;                                   // the same for all threads
      const int be = __double2hiint(ss) >> 20;      // biased exponent: |v|^2 in 2^(+-700)
      if (be < 323 || be > 1723) ss = scale_column(v, j, n, ss, red, ex);
      if (warp == 0) {
        const double x0 = v[j + 1];
        const double nrm = ss > 0.0 ? ss * fast_rsqrt(ss) : 0.0;
        const double alpha = x0 >= 0.0 ? -nrm : nrm;
        // |v|^2 / 2 = |x|^2 + |x0| |x|
        const double h = fma(fabs(x0), nrm, ss);
        const double t = h > 0.0 ? fast_inv(h) : 0.0;
        __syncwarp();
        if (lane == 0) {
          v[j + 1] = x0 - alpha;
          s_tau = t;
          if (q == 0) {
            const double ej = h > 0.0 ? alpha : x0;
            e[j] = ex ? ldexp(ej, ex) : ej;
            tau[j] = t;
          }
        }
      }
    }
    __syncthreads();
    const double tj = s_tau;
    double* pj = pb + (j & 1) * n;
    double* cj = cb + (j & 1) * n;
    const int i0 = j + 1 <= q ? 0 : (j + 1 - q + C - 1) / C;
    for (int i = i0 + warp; i < nloc; i += kTrWarps) {
      const int r = q + i * C;
      double* row = SM ? rows + (int64_t)i * n : A + (int64_t)r * n;
      const double vr = vprev[r], wr = wp[r];
      double acc0 = 0.0, acc1 = 0.0, first = 0.0;
      int c = j + 1 + lane;
      for (; c + 32 < n; c += 64) {
        double b0 = row[c], b1 = row[c + 32];
        b0 = fma(-vr, wp[c], b0);
        b1 = fma(-vr, wp[c + 32], b1);
        b0 = fma(-wr, vprev[c], b0);
        b1 = fma(-wr, vprev[c + 32], b1);
        row[c] = b0;
        row[c + 32] = b1;
        acc0 = fma(b0, v[c], acc0);
        acc1 = fma(b1, v[c + 32], acc1);
        if (c == j + 1) first = b0;
      }
      if (c < n) {
        double b0 = row[c];
        b0 = fma(-vr, wp[c], b0);
        b0 = fma(-wr, vprev[c], b0);
        row[c] = b0;
        acc0 = fma(b0, v[c], acc0);
        if (c == j + 1) first = b0;
      }
      const double p = tj * warp_sum(acc0 + acc1);
      first = __shfl_sync(0xffffffffu, first, 0);
      if (lane < C) {
        *cl.map_shared_rank(pj + r, lane) = p;
        *cl.map_shared_rank(cj + r, lane) = first;
      }
    }
    cl.sync();
    if (warp < kVecWarps) {
      double vp = 0.0;
      for (int r = j + 1 + tid; r < n; r += kVecWarps * 32) vp = fma(v[r], pj[r], vp);
      vp = vec_sum(vp, red[1]);
      const double K = 0.5 * tj * vp;
      const double v1 = v[j + 1], w1 = fma(-K, v1, pj[j + 1]);
      for (int r = j + 1 + tid; r < n; r += kVecWarps * 32) {
        const double w = fma(-K, v[r], pj[r]);
        wp[r] = w;
        if (r > j + 1) vprev[r] = fma(-w, v1, fma(-v[r], w1, cj[r]));     // x_{j+1}
      }
      if (q == 0 && tid == 0) d[j + 1] = fma(-2.0 * v1, w1, cj[j + 1]);
      asm volatile("bar.sync 1, %0;" ::"n"(kVecWarps * 32) : "memory");
    } else if (q == j % C) {
      for (int r = j + 1 + tid - kVecWarps * 32; r < n; r += kTrThreads - kVecWarps * 32)
        Vr[r + (int64_t)j * n] = v[r];
    }
  }
  __syncthreads();
  // the last entries: e[n-2] = x_{n-2}, d[n-1] with the last update applied
  const int jl = n - 3;                             // last column reduced (n >= 3)
  if (tid == 0) {
    if (q == 0) {
      if (n == 2) e[0] = A[1];
      if (n >= 3) e[n - 2] = ((n - 2) & 1 ? V1 : V0)[n - 1];
      e[n - 1] = 0.0;
      tau[n - 1] = 0.0;
      if (n >= 2) tau[n - 2] = 0.0;
    }
    if (n >= 2 && q == (n - 1) % C) {
      const double b = SM ? rows[(int64_t)((n - 1) / C) * n + n - 1] : A[(int64_t)(n - 1) * n + n - 1];
      const double* vl = (jl & 1) ? V1 : V0;
      d[n - 1] = n >= 3 ? fma(-2.0 * vl[n - 1], wp[n - 1], b) : b;
    }
  }
  cl.sync();
}

// Eigenvalues of T below x: sign changes of the Sturm polynomials
// p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}, whose chain is one FMA a step
// (the quotient form's is a division).  T is scaled to at most 1; p is rescaled
// by powers of two every four steps, within which it cannot leave the FP64
// range (the points stay above 1e-60).  A zero counts as an infinitesimal of
// the other sign, as the quotient form's guard has it: the four steps are then
// done again with the test after each.
__device__ __forceinline__ bool is_zero(double x) {
  return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}

__device__ __forceinline__ int sturm_count(const double* d, const double* e2, int n, double x) {
  int cnt = 0;
  double p0 = 1.0, p1 = d[0] - x;
  if (is_zero(p1)) p1 = -1e-100;
  cnt += __double2hiint(p1) < 0;
  for (int i0 = 1; i0 < n; i0 += 4) {
    // the larger exponent of the two to 0
    const int h = max(__double2hiint(p0) & 0x7ff00000, __double2hiint(p1) & 0x7ff00000);
    const double s = __hiloint2double(0x7fe00000 - h, 0);
    p0 *= s;
    p1 *= s;
    double q0 = p0, q1 = p1;
    int c4 = 0;
    bool zero = false;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u;
      if (i < n) {
        const double t = e2[i - 1] * q0;
        q0 = q1;
        q1 = fma(d[i] - x, q1, -t);
        zero |= is_zero(q1);
        c4 += (__double2hiint(q1) ^ __double2hiint(q0)) < 0;
      }
    }
    if (zero) {
      q0 = p0;
      q1 = p1;
      c4 = 0;
      for (int i = i0; i < min(n, i0 + 4); ++i) {
        const double t = e2[i - 1] * q0;
        q0 = q1;
        q1 = fma(d[i] - x, q1, -t);
        if (is_zero(q1)) {
          q0 = copysign(1.0, q0);
          q1 = -q0 * 1e-100;
        }
        c4 += (__double2hiint(q1) ^ __double2hiint(q0)) < 0;
      }
    }
    cnt += c4;
    p0 = q0;
    p1 = q1;
  }
  return cnt;
}

// Stage 2: eigenvalue b (descending order) per CTA.  Four warps, one for each
// of the SM's FP64 pipes, try 128 points a round: 8 rounds.  Bound by those
// pipes, three operations a point and step.  n = 360, 72 eigenvalues: 2.6 -> 0.65 ms.
constexpr int kSectWarps = 4;

__global__ void __launch_bounds__(32 * kSectWarps) k_tridiag_multisect(
    const double* __restrict__ d, const double* __restrict__ e, int n, double* __restrict__ w) {
  extern __shared__ double sm[];
  double* sd = sm;
  double* se2 = sm + n;
  __shared__ unsigned above[2][kSectWarps];
  __shared__ double s_lo[kSectWarps], s_hi[kSectWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = blockIdx.x;
  double lo = 1e300, hi = -1e300;
  for (int i = tid; i < n; i += 32 * kSectWarps) {
    const double rad = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - rad);
    hi = fmax(hi, d[i] + rad);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  for (int v = 0; v < kSectWarps; ++v) {
    lo = fmin(lo, s_lo[v]);
    hi = fmax(hi, s_hi[v]);
  }
  if (lo == 0.0 && hi == 0.0) {                 // T = 0
    if (tid == 0) w[b] = 0.0;
    return;
  }
  // T scaled by a power of two to at most 1 (exact)
  int ex = 0;
  frexp(fmax(fabs(lo), fabs(hi)), &ex);
  const double sc = ldexp(1.0, -max(-1000, min(1000, ex)));
  for (int i = tid; i < n; i += 32 * kSectWarps) {
    sd[i] = d[i] * sc;
    const double es = (i + 1 < n) ? e[i] * sc : 0.0;
    se2[i] = es * es;
  }
  lo *= sc;
  hi *= sc;
  __syncthreads();
  const double pad = 4.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + 1e-300;
  lo -= pad;
  hi += pad;
  const int target = n - 1 - b;                 // ascending index
  constexpr int kPoints = 32 * kSectWarps;
  for (int round = 0; round < 28; ++round) {     // 129^-28 > 1e-60
    if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + 1e-300) break;
    auto point = [&](int k) { return lo + (hi - lo) * ((double)(k + 1) * (1.0 / (kPoints + 1))); };
    const int cnt = sturm_count(sd, se2, n, point(tid));
    const unsigned m = __ballot_sync(0xffffffffu, cnt > target);
    if (lane == 0) above[round & 1][warp] = m;
    __syncthreads();
    int L = kPoints;                            // first point above the target
    for (int v = kSectWarps - 1; v >= 0; --v)
      if (above[round & 1][v]) L = 32 * v + __ffs(above[round & 1][v]) - 1;
    const double nlo = L > 0 ? point(L - 1) : lo;
    if (L < kPoints) hi = point(L);
    lo = nlo;
  }
  if (tid == 0) w[b] = 0.5 * (lo + hi) / sc;
}

// Stage 3: eigenvector b by one warp: inverse iteration on T (one lane, the
// LU factors once, three solves), then u = Q z with z in registers, NPL
// elements a lane, so a reflector costs one warp sum and no CTA barrier
// (n = 360: 1.9 -> 1.0 ms).  Dynamic shared memory: 7 n doubles, n bytes.
template <int NPL>
__global__ void __launch_bounds__(32) k_tridiag_vectors(
    const double* __restrict__ d, const double* __restrict__ e, const double* __restrict__ tau,
    const double* __restrict__ Vr, const double* __restrict__ w, int n, double* __restrict__ U) {
  extern __shared__ double sm[];
  double* sd = sm;
  double* se = sd + n;
  double* dg = se + n;         // pivots, then their reciprocals
  double* u1 = dg + n;
  double* u2 = u1 + n;
  double* ml = u2 + n;         // multipliers
  double* z = ml + n;
  unsigned char* sw = reinterpret_cast<unsigned char*>(z + n);   // rows swapped
  const int lane = threadIdx.x, b = blockIdx.x;
  double tn = 0.0;
  for (int i = lane; i < n; i += 32) {
    sd[i] = d[i];
    se[i] = e[i];
    tn = fmax(tn, fabs(d[i]) + fabs(e[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0));
  }
  for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
  // separate (nearly) equal eigenvalues: w is descending, and s_i = s_{i-1} - pert
  // where s_{i-1} - w_i < pert, else w_i.  s_i >= w_i - i pert, so a gap of
  // (i + 1) pert resets the chain: it starts at the last such gap up to b.
  const double pert = 10.0 * DBL_EPSILON * tn + 1e-300;
  int start = 0;
  for (int top = b; top > 0; top -= 32) {
    const int i = top - lane;
    const bool gap = i > 0 && w[i - 1] - w[i] >= (double)(i + 1) * pert;
    const unsigned m = __ballot_sync(0xffffffffu, gap);
    if (m) {
      start = top - (__ffs(m) - 1);
      break;
    }
  }
  double lam = w[start];
  for (int i = start + 1; i <= b; ++i) {
    const double wi = w[i];
    lam = (lam - wi < pert) ? lam - pert : wi;
  }
  __syncwarp();
  if (lane == 0) {
    uint32_t seed = 0x9e3779b9u * (uint32_t)(b + 1);
    for (int i = 0; i < n; ++i) {
      seed = seed * 1664525u + 1013904223u;
      z[i] = 0.5 + (double)(seed >> 8) * (1.0 / 16777216.0);
    }
    double a = sd[0] - lam, bb = (n > 1 ? se[0] : 0.0), c = 0.0;
    for (int i = 0; i + 1 < n; ++i) {
      const double sub = se[i];
      const double na = sd[i + 1] - lam, nb = (i + 2 < n ? se[i + 1] : 0.0);
      if (fabs(a) >= fabs(sub)) {
        const double mlt = (a != 0.0 ? fast_div(sub, a) : 0.0);
        dg[i] = a; u1[i] = bb; u2[i] = c; ml[i] = mlt; sw[i] = 0;
        a = fma(-mlt, bb, na); bb = fma(-mlt, c, nb); c = 0.0;
      } else {
        const double mlt = fast_div(a, sub);
        dg[i] = sub; u1[i] = na; u2[i] = nb; ml[i] = mlt; sw[i] = 1;
        a = fma(-mlt, na, bb); bb = fma(-mlt, nb, c); c = 0.0;
      }
    }
    dg[n - 1] = a;
  }
  __syncwarp();
  const double guard = DBL_EPSILON * tn + 1e-300;
  for (int i = lane; i < n; i += 32) {
    const double p = dg[i];
    dg[i] = 1.0 / (fabs(p) > guard ? p : (p >= 0.0 ? guard : -guard));
    if (i + 1 >= n) u1[i] = 0.0;
    if (i + 2 >= n) u2[i] = 0.0;
  }
  __syncwarp();
  for (int pass = 0; pass < 3; ++pass) {
    if (lane == 0) {
      double zc = z[0];
#pragma unroll 4
      for (int i = 0; i + 1 < n; ++i) {
        const double zn = z[i + 1], mm = ml[i];
        const bool swap = sw[i] != 0;
        const double up = swap ? zn : zc, dn = swap ? zc : zn;
        z[i] = up;
        zc = fma(-mm, up, dn);
      }
      double z1 = zc * dg[n - 1], z2 = 0.0;
      z[n - 1] = z1;
#pragma unroll 4
      for (int i = n - 2; i >= 0; --i) {
        const double t = fma(-u2[i], z2, z[i]);
        z2 = z1;
        z1 = fma(-u1[i], z1, t) * dg[i];
        z[i] = z1;
      }
    }
    __syncwarp();
    double nrm = 0.0;
    for (int i = lane; i < n; i += 32) nrm = fmax(nrm, fabs(z[i]));
    for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
    const double inv = 1.0 / nrm;
    for (int i = lane; i < n; i += 32) z[i] *= inv;
    __syncwarp();
  }
  // u = H_0 H_1 ... H_{n-3} z
  double y[NPL];
#pragma unroll
  for (int v = 0; v < NPL; ++v) y[v] = lane + 32 * v < n ? z[lane + 32 * v] : 0.0;
  auto load = [&](int j, double* x) {
#pragma unroll
    for (int v = 0; v < NPL; ++v) {
      const int r = lane + 32 * v;
      x[v] = r > j && r < n ? __ldg(Vr + r + (int64_t)j * n) : 0.0;
    }
  };
  auto apply = [&](int j, const double* x) {
    double t0 = 0.0, t1 = 0.0;
#pragma unroll
    for (int v = 0; v < NPL; ++v) {
      if (32 * v + 31 > j) {
        if (v & 1) t1 = fma(x[v], y[v], t1);
        else t0 = fma(x[v], y[v], t0);
      }
    }
    const double dot = -warp_sum(t0 + t1) * __ldg(tau + j);
#pragma unroll
    for (int v = 0; v < NPL; ++v)
      if (32 * v + 31 > j) y[v] = fma(dot, x[v], y[v]);
  };
  if constexpr (NPL <= 24) {       // the next reflector is loaded under this one
    double xa[NPL], xb[NPL];
    if (n >= 3) load(n - 3, xa);
    for (int j = n - 3; j >= 0; j -= 2) {
      if (j > 0) load(j - 1, xb);
      apply(j, xa);
      if (j > 1) load(j - 2, xa);
      if (j > 0) apply(j - 1, xb);
    }
  } else {                          // many vectors an SM instead
    double xa[NPL];
    for (int j = n - 3; j >= 0; --j) {
      load(j, xa);
      apply(j, xa);
    }
  }
  double nn = 0.0;
#pragma unroll
  for (int v = 0; v < NPL; ++v) nn = fma(y[v], y[v], nn);
  nn = warp_sum(nn);
  const double inv = 1.0 / sqrt(nn);
#pragma unroll
  for (int v = 0; v < NPL; ++v)
    if (lane + 32 * v < n) U[(int64_t)b * n + lane + 32 * v] = y[v] * inv;
}

// N = (3 I - S) / 2; *dev = max |S - I| (FP64 bits, zeroed before)
__global__ void __launch_bounds__(256) k_newton_schulz(const double* __restrict__ S,
                                                       double* __restrict__ N, int r,
                                                       unsigned long long* dev) {
  const int64_t total = (int64_t)r * r;
  double m = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double one = (i % r == i / r) ? 1.0 : 0.0, s = S[i];
    const double dv = fabs(s - one);
    m = dv > m || dv != dv ? dv : m;             // a NaN stays
    N[i] = 1.5 * one - 0.5 * s;
  }
  unsigned long long mb = (unsigned long long)__double_as_longlong(m);
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, mb, o);
    mb = t > mb ? t : mb;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(dev, mb);
}

// Fallback orthonormalisation: classical Gram-Schmidt with one
// reorthogonalisation pass, column by column, one CTA.
__global__ void __launch_bounds__(1024) k_cgs2(double* __restrict__ U, int n, int r,
                                               double* __restrict__ coef) {
  __shared__ double red[32];
  for (int j = 0; j < r; ++j) {
    double* uj = U + (int64_t)j * n;
    for (int pass = 0; pass < 2; ++pass) {
      // coef[i] = u_i . u_j for i < j: one warp per i
      for (int i = threadIdx.x >> 5; i < j; i += blockDim.x >> 5) {
        const double* ui = U + (int64_t)i * n;
        double s = 0.0;
        for (int t = threadIdx.x & 31; t < n; t += 32) s += ui[t] * uj[t];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) coef[i] = s;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < n; t += blockDim.x) {
        double s = uj[t];
        for (int i = 0; i < j; ++i) s -= coef[i] * U[(int64_t)i * n + t];
        uj[t] = s;
      }
      __syncthreads();
    }
    double nn = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) nn += uj[t] * uj[t];
    nn = cta_sum(nn, red);
    const double inv = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) uj[t] *= inv;
    __syncthreads();
  }
}

__global__ void k_symmetrize_lower(double* A, int n) {
  const int64_t total = (int64_t)n * n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i % n), c = (int)(i / n);
    if (r > c) {
      const double s = 0.5 * (A[i] + A[c + (int64_t)r * n]);
      A[i] = s;
      A[c + (int64_t)r * n] = s;
    }
  }
}

}  // namespace

namespace {

// Cluster size and shared memory of the tridiagonalisation: 16 CTAs (a
// non-portable size) from n = 128 on where the device can hold them, else 8;
// rows in shared memory if they fit.
struct TriPlan {
  int cluster;
  bool sm;
  size_t smem;
};

template <bool SM>
ttg_status tri_launch(const TriPlan& P, cudaStream_t st, double* A, int n, double* d, double* e,
                      double* tau, double* Vr, bool probe, int* fits) {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_tridiag_cluster<SM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kTrMaxSmem);
    if (attr == cudaSuccess)
      attr = cudaFuncSetAttribute(k_tridiag_cluster<SM>,
                                  cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
  if (attr != cudaSuccess) return TTG_CUDA_ERR;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)P.cluster);
  cfg.blockDim = dim3(kTrThreads);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)P.cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (probe) {
    *fits = 0;
    if (cudaOccupancyMaxActiveClusters(fits, k_tridiag_cluster<SM>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      *fits = 0;
    }
    return TTG_OK;
  }
  TTG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_tridiag_cluster<SM>, A, n, d, e, tau, Vr));
  TTG_COUNT();
  return TTG_OK;
}

ttg_status tridiagonalise(cudaStream_t st, double* A, int n, double* d, double* e, double* tau,
                          double* Vr) {
  const size_t vec = (size_t)7 * n * sizeof(double);
  const int sizes[2] = {kMaxCluster, 8};
  for (int t = n >= 128 ? 0 : 1; t < 2; ++t) {
    TriPlan P{sizes[t], true, 0};
    P.smem = vec + (size_t)((n + P.cluster - 1) / P.cluster) * n * sizeof(double);
    if (P.smem > kTrMaxSmem) {
      P.sm = false;
      P.smem = vec;
    }
    if (P.cluster > 8) {
      int fits = 0;
      TTG_TRY(P.sm ? tri_launch<true>(P, st, A, n, d, e, tau, Vr, true, &fits)
                   : tri_launch<false>(P, st, A, n, d, e, tau, Vr, true, &fits));
      if (fits < 1) continue;
    }
    return P.sm ? tri_launch<true>(P, st, A, n, d, e, tau, Vr, false, nullptr)
                : tri_launch<false>(P, st, A, n, d, e, tau, Vr, false, nullptr);
  }
  return TTG_CUDA_ERR;
}

template <int NPL>
ttg_status vectors_launch(cudaStream_t st, const double* d, const double* e, const double* tau,
                          const double* Vr, const double* w, int n, int r, double* U) {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_tridiag_vectors<NPL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (7 * (int)sizeof(double) + 1) * 32 * NPL);
  });
  if (attr != cudaSuccess) return TTG_CUDA_ERR;
  k_tridiag_vectors<NPL><<<r, 32, (7 * sizeof(double) + 1) * n, st>>>(d, e, tau, Vr, w, n, U); TTG_COUNT();
  return cudaGetLastError() == cudaSuccess ? TTG_OK : TTG_CUDA_ERR;
}

}  // namespace

ttg_status sym_topk(ttg_op* op, double* A, int n, int r, double* w, double* U, int* d_status) {
  if (r < 1 || r > n || n > kMaxN) return TTG_BAD_ARG;
  const int64_t nn = (int64_t)n * n;
  const size_t need = (size_t)(nn + 3 * (int64_t)n + 2 * (int64_t)r * r + (int64_t)n * r + 64) *
                      sizeof(double);
  if (op->eigbuf.bytes < need) TTG_TRY(op->eigbuf.alloc(need));
  cudaStream_t st = op->stream;
  double* Vr = op->eigbuf.as<double>();
  double* dd = Vr + nn;
  double* ee = dd + n;
  double* tt = ee + n;
  double* S = tt + n;
  double* Li = S + (int64_t)r * r;
  double* U2 = Li + (int64_t)r * r;
  unsigned long long* dev = reinterpret_cast<unsigned long long*>(U2 + (int64_t)n * r);
  k_symmetrize_lower<<<64, 256, 0, st>>>(A, n); TTG_COUNT();
  TTG_LAUNCHED(op);
  TTG_TRY(tridiagonalise(st, A, n, dd, ee, tt, Vr));
  TTG_LAUNCHED(op);
  k_tridiag_multisect<<<r, 32 * kSectWarps, 2 * n * sizeof(double), st>>>(dd, ee, n, w); TTG_COUNT();
  TTG_LAUNCHED(op);
  if (n <= 128) TTG_TRY(vectors_launch<4>(st, dd, ee, tt, Vr, w, n, r, U));
  else if (n <= 256) TTG_TRY(vectors_launch<8>(st, dd, ee, tt, Vr, w, n, r, U));
  else if (n <= 384) TTG_TRY(vectors_launch<12>(st, dd, ee, tt, Vr, w, n, r, U));
  else if (n <= 768) TTG_TRY(vectors_launch<24>(st, dd, ee, tt, Vr, w, n, r, U));
  else if (n <= 1280) TTG_TRY(vectors_launch<40>(st, dd, ee, tt, Vr, w, n, r, U));
  else TTG_TRY(vectors_launch<64>(st, dd, ee, tt, Vr, w, n, r, U));
  TTG_LAUNCHED(op);
  const DOp Ut{U, (int64_t)n, 1, 0}, Un{U, 1, (int64_t)n, 0};
  // U^T U and U M (M r x r, M(k, j) at M[k ks + j js]): on the tensor cores from
  // 1e8 flops on, else double-FP32.  All pairs of n = 200 there 2,042 us, here
  // 2,014; n = 368 5,009 and 5,006; n = 450 7,349 and 7,468; n = 1,200 73.1 and 75.3 ms.
  const bool big = 2.0 * n * r * r >= 1e8;
  const OzOperand cols{U, r, n, n, 1}, urows{U, n, r, 1, n};
  auto gram = [&]() -> ttg_status {
    if (big && ozgemm_supported(cols, cols)) {
      const ttg_status s = ozgemm(op, cols, cols, S, OzLayout{1, r}, true);
      if (s != TTG_OOM) return s;
    }
    return dgemm(st, r, r, n, 1, Ut, Un, S, 1, r, 0, op->partial);
  };
  auto product = [&](const double* M, int64_t ks, int64_t js) -> ttg_status {
    const OzOperand B{M, r, r, js, ks};
    if (big && ozgemm_supported(urows, B)) {
      const ttg_status s = ozgemm(op, urows, B, U2, OzLayout{1, n}, false);
      if (s != TTG_OOM) return s;
    }
    return dgemm(st, n, r, r, 1, Un, DOp{M, ks, js, 0}, U2, 1, n, 0, op->partial);
  };
  // S = U^T U = I + E; Li = (3 I - S) / 2
  TTG_TRY(gram());
  TTG_CUDA_TRY(cudaMemsetAsync(dev, 0, 8, st));
  k_newton_schulz<<<32, 256, 0, st>>>(S, Li, r, dev); TTG_COUNT();
  TTG_LAUNCHED(op);
  double far = 0.0;
  TTG_CUDA_TRY(cudaMemcpyAsync(&far, dev, 8, cudaMemcpyDeviceToHost, st));
  TTG_CUDA_TRY(cudaMemsetAsync(d_status, 0, 4, st));
  TTG_CUDA_TRY(cudaStreamSynchronize(st));
  if (far <= 1e-8) {
    TTG_TRY(product(Li, 1, r));
    TTG_CUDA_TRY(cudaMemcpyAsync(U, U2, (size_t)n * r * sizeof(double), cudaMemcpyDeviceToDevice,
                                 st));
    op->launches += 2;
    return TTG_OK;
  }
  // Cholesky QR2: U <- U L^-T with U^T U = L L^T
  for (int pass = 0; pass < 2; ++pass) {
    if (pass > 0) TTG_TRY(gram());
    TTG_TRY(cholesky_inv(op, S, Li, r, d_status));
    int stat = 0;
    TTG_CUDA_TRY(cudaMemcpyAsync(&stat, d_status, 4, cudaMemcpyDeviceToHost, st));
    TTG_CUDA_TRY(cudaStreamSynchronize(st));
    if (stat != 0) {
      k_cgs2<<<1, 1024, 0, st>>>(U, n, r, S); TTG_COUNT();
      TTG_LAUNCHED(op);
      TTG_CUDA_TRY(cudaMemsetAsync(d_status, 0, 4, st));
      break;
    }
    TTG_TRY(product(Li, r, 1));
    TTG_CUDA_TRY(cudaMemcpyAsync(U, U2, (size_t)n * r * sizeof(double), cudaMemcpyDeviceToDevice,
                                 st));
    op->launches += 4;
  }
  return TTG_OK;
}

}  // namespace ttg
