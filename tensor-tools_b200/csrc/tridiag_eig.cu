// Two-phase symmetric eigensolver for the per-QN-sector density matrices of
// the block SVD (qtensor/qtensor_op.cpp:1229-1300): all eigenvalues first (so
// the host can apply the truncation rule of :1290-1300), then eigenvectors
// only for the states that are kept.
//
// Phase 1 (tt_sym_eigvals_batched): Householder reduction to tridiagonal form
//   T = Q^T G Q (Golub & Van Loan, "Matrix Computations", 4th ed., alg. 8.3.1),
//   reflectors kept below the subdiagonal of G -- sectors with n <= SN by one
//   CTA each with the matrix in shared memory, larger ones by a cluster of CTAs;
//   then every eigenvalue of every T by bisection on Sturm sequence counts
//   (ibid. sec. 8.4.1), spread over the GPU.
// Phase 2 (tt_sym_eigvecs_batched): inverse iteration on T - lambda I
//   (tridiagonal LU with partial pivoting, tiny pivots replaced by eps*||T||),
//   orthogonalisation inside clusters of close eigenvalues (gap <= 1e-3 ||T||,
//   the clustering rule of LAPACK's inverse iteration) and back-transformation
//   z = Q y with the stored reflectors -- one CTA per sector with n <= SN, GPU-wide
//   kernels batched over the larger ones.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "tt_internal.h"

namespace {

constexpr int TT = 512;          // threads per CTA
constexpr int SN = 128;          // sectors up to this size: one CTA, matrix in shared memory
constexpr int SB = SN / 32;      // row chunks of 32 of such a sector
constexpr int MAX_N = 4096;
constexpr int INV_ITERS = 3;

struct EigDev {
  int64_t g_off, w_off, a_off;
  int32_t n, flags, nvec, nb;  // nb: panel width of the blocked reduction
  int64_t s_off;               // its place in the scratch of the cluster reductions
};

__device__ double block_reduce(double v, double* red, bool is_max) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double u = __shfl_down_sync(0xffffffffu, v, o);
    v = is_max ? fmax(v, u) : v + u;
  }
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = red[0];
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) s = is_max ? fmax(s, red[i]) : s + red[i];
    red[32] = s;
  }
  __syncthreads();
  return red[32];
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// number of eigenvalues of T that are < x: the sign changes of the Sturm
// sequence p_i = (d_i - x) p_{i-1} - e2_{i-1} p_{i-2} of leading principal
// minors (Golub & Van Loan, "Matrix Computations", 4th ed., sec. 8.4.1).
// de[i] = (d_i, e2_{i-1}) of T scaled to a norm in [1/2, 1), padded to a
// multiple of 8 with (4, 0), which keep the sign.  Off-diagonals are floored at
// 2^-60 (their squares at STURM_E2), far below the rounding of T, so a vanishing
// minor is followed by one of the opposite sign of the one before it and needs
// no test of its own; a step then is one dependent FMA, and the pair (p_{i-1},
// p_i), which shrinks by at most 2^-480 and grows by at most 3^8 over 8 steps,
// is rescaled by a power of two every 8 steps when it has left 2^+-300.
constexpr double STURM_E2 = 0x1p-120;
__device__ __forceinline__ int sturm_count(const double2* de, int npad, double x) {
  double pm = 0.0, p = 1.0;
  int c = 0;
  for (int i = 0; i < npad; i += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const double2 t = de[i + u];
      const double pn = fma(t.x - x, p, -(t.y * pm));
      c += (unsigned)(__double2hiint(pn) ^ __double2hiint(p)) >> 31;
      pm = p;
      p = pn;
    }
    const int ex = max(__double2hiint(p) & 0x7fffffff, __double2hiint(pm) & 0x7fffffff) >> 20;
    if (ex > 1023 + 300 || ex < 1023 - 300) {
      const double sc = __hiloint2double((2046 - ex) << 20, 0);
      p *= sc;
      pm *= sc;
    }
  }
  return c;
}

// ---------------------------------------------------------------------------
// Sectors with n <= SN: tridiagonalisation by one CTA, matrix in shared memory.
//
// A column costs two barriers.  Every warp forms the reflector v of column k
// for itself (same data, same order: rows lane + 32 b in registers, a private
// copy in shared memory for the column factors), then takes its share of the
// trailing columns in one pass that applies the previous reflector's rank-2
// update and accumulates A22 v of the new one, so the matrix is read and
// written once per column.  After barrier 1 thread r sums row r of A22 v over
// the warps; after barrier 2 every warp forms w on its own rows.
//
// Bound by the latency of that chain (square root, two reciprocals, two warp
// sums, two barriers: 1.5 us a column), not by its shared-memory traffic.
// Measured with the eigenvalues by the kernel below, against five barriers a
// column, indices by division and a bisection per CTA: a block SVD at bond
// dimension 75 (n <= 36) 153 -> 54 + 22 us, at 512 (n <= 75) 385 -> 127 us.  It
// stops at 128: its working arrays and a 128 x 128 matrix take 197 KB.
// doubles of shared memory
__host__ __device__ constexpr int64_t small_smem(int n, int nw) { return (int64_t)n * n + 4 * (int64_t)nw * n + n; }
// six sectors of 20 and of 32 states: 58 and 74 us with 256 threads, 64 and 85 with 512
constexpr int small_threads(int nmax) { return nmax <= 32 ? 256 : 512; }

__global__ void __launch_bounds__(TT, 1)
tridiag_small(const EigDev* __restrict__ probs, double* G, double* Tg, double* W, const double* Amat) {
  extern __shared__ double sm[];
  __shared__ double dots[SB], red[33];
  // the cluster kernel that may follow reads nothing of this one's
  asm volatile("griddepcontrol.launch_dependents;");
  const EigDev P = probs[blockIdx.x];
  const int n = P.n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  if (n <= 0) return;
  if (P.flags & TT_EIG_ROW_1X2) {
    if (tid == 0) {
      const double a = Amat[P.a_off], b = Amat[P.a_off + 1];
      W[P.w_off] = a * a + b * b;
      W[P.w_off + 1] = 0.0;
    }
    return;
  }
  double* dg = Tg + 3 * P.w_off;  // d[n], e[n], tau[n]
  double* eg = dg + n;
  double* tg = eg + n;
  double* Gp = G + P.g_off;
  double* A = sm;                            // [n][n]
  double* part = A + n * n;                  // [nw][n]: A22 v by warp
  double* vold = part + nw * n + warp * n;   // this warp's copies: the previous v,
  double* vnew = vold + nw * n;              // the new one,
  double* wold = vnew + nw * n;              // and the previous w
  double* ps = part + 4 * nw * n;            // [n]: p = tau A22 v
  // squares of the entries must neither overflow nor vanish: a matrix far from
  // 1 is scaled by a power of two (T is scaled back; the reflectors do not care)
  double amax = 0.0;
  for (int i = tid; i < n * n; i += blockDim.x) {
    const double g = Gp[i];
    A[i] = g;
    amax = fmax(amax, fabs(g));
  }
  for (int i = lane; i < n; i += 32) vold[i] = wold[i] = 0.0;
  amax = block_reduce(amax, red, true);
  double isc = 1.0;
  if (amax > 0.0 && isfinite(amax) && (amax < 0x1p-300 || amax > 0x1p300)) {
    int ex;
    frexp(amax, &ex);
    ex = max(ex, -1000);
    isc = ldexp(1.0, ex);
    for (int i = tid; i < n * n; i += blockDim.x) A[i] = ldexp(A[i], -ex);
  }
  double vo[SB], wo[SB];  // the previous v, w on the rows lane + 32 b
#pragma unroll
  for (int b = 0; b < SB; ++b) vo[b] = wo[b] = 0.0;
  __syncthreads();
  for (int k = 0; k + 2 < n; ++k) {
    // column k as the previous reflector leaves it, and its own reflector
    const double vk = vold[k], wk = wold[k];
    double x[SB], sig = 0.0;
#pragma unroll
    for (int b = 0; b < SB; ++b) {
      const int r = lane + 32 * b;
      x[b] = 0.0;
      if (r >= k && r < n) x[b] = A[r + n * k] - vo[b] * wk - wo[b] * vk;
      if (r >= k + 2) sig += x[b] * x[b];
    }
    const double sigma = warp_sum(sig);
    auto row = [&](int i) {  // x of row i, to every lane
      double t = x[0];
#pragma unroll
      for (int b = 1; b < SB; ++b)
        if ((i >> 5) == b) t = x[b];
      return __shfl_sync(0xffffffffu, t, i & 31);
    };
    const double dk = row(k), alpha = row(k + 1);
    double tau = 0.0, beta = alpha, scale = 0.0;
    if (sigma != 0.0) {
      const double mu = sqrt(alpha * alpha + sigma);
      beta = alpha <= 0.0 ? mu : -mu;
      tau = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
    }
    double vn[SB], pr[SB];
#pragma unroll
    for (int b = 0; b < SB; ++b) {
      const int r = lane + 32 * b;
      vn[b] = r == k + 1 ? 1.0 : (r >= k + 2 ? x[b] * scale : 0.0);
      pr[b] = 0.0;
      if (r < n) vnew[r] = vn[b];
    }
    __syncwarp();
    for (int c = k + 1 + warp; c < n; c += nw) {
      const double vc = vold[c], wc = wold[c], nc = vnew[c];
      double* col = A + n * c;
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int r = lane + 32 * b;
        if (r > k && r < n) {
          const double t = fma(-wo[b], vc, fma(-vo[b], wc, col[r]));
          col[r] = t;
          pr[b] = fma(t, nc, pr[b]);
        }
      }
    }
#pragma unroll
    for (int b = 0; b < SB; ++b)
      if (lane + 32 * b < n) part[warp * n + lane + 32 * b] = pr[b];
    __syncthreads();  // 1
    if (warp < SB) {
      double p = 0.0, v = 0.0;
      if (tid > k && tid < n) {
        for (int w = 0; w < nw; ++w) p += part[w * n + tid];
        p *= tau;
        v = vnew[tid];
        ps[tid] = p;
      }
      const double d = warp_sum(v * p);
      if (lane == 0) dots[warp] = d;
    }
    if (warp == nw - 1) {  // the reflector, for phase 2, and T
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int r = lane + 32 * b;
        if (r >= k + 2 && r < n) A[r + n * k] = vn[b];
      }
      if (lane == 0) {
        dg[k] = dk * isc;
        eg[k] = beta * isc;
        tg[k] = tau;
      }
    }
    __syncthreads();  // 2
    double K = dots[0];
#pragma unroll
    for (int b = 1; b < SB; ++b) K += dots[b];
    K *= 0.5 * tau;
#pragma unroll
    for (int b = 0; b < SB; ++b) {
      const int r = lane + 32 * b;
      vo[b] = vn[b];
      wo[b] = r > k && r < n ? ps[r] - K * vn[b] : 0.0;
      if (r < n) wold[r] = wo[b];
    }
    double* t = vold;
    vold = vnew;
    vnew = t;
    __syncwarp();
  }
  __syncthreads();
  if (tid == 0) {  // the last 2 x 2 block
    const int i = n - 2, j = n - 1;
    if (n >= 2) {
      dg[i] = (A[i + n * i] - 2.0 * vold[i] * wold[i]) * isc;
      eg[i] = (A[j + n * i] - vold[j] * wold[i] - wold[j] * vold[i]) * isc;
      tg[i] = 0.0;
    }
    dg[j] = (A[j + n * j] - 2.0 * vold[j] * wold[j]) * isc;
    eg[j] = 0.0;
    tg[j] = 0.0;
  }
  for (int i = tid; i < n * n; i += blockDim.x) Gp[i] = A[i];
}

// solve (T - lambda I) y = b in place (y holds b on entry); U holds 3n scratch
// The LU factors go to u0, u1, u2, entry i at [i * ustride] (ustride > 1
// interleaves the factors of neighbouring threads, so that their accesses
// coalesce); y's entry i is at [i * ystride].
__device__ void tri_solve(const double* d, const double* e, int n, double lambda, double tiny, double* y,
                          double* u0, double* u1, double* u2, int ystride, int ustride) {
  // forward elimination with partial pivoting, transforming b on the fly
  double di = d[0] - lambda, si = n > 1 ? e[0] : 0.0, ti = 0.0;
  double bi = y[0];
  for (int i = 0; i + 1 < n; ++i) {
    double ci = e[i];
    double an = d[i + 1] - lambda;
    double bn = (i + 2 < n) ? e[i + 1] : 0.0;
    double bnext = y[(int64_t)(i + 1) * ystride];
    if (fabs(di) >= fabs(ci)) {
      if (di == 0.0) di = tiny;
      double mlt = ci / di;
      u0[(int64_t)i * ustride] = di;
      u1[(int64_t)i * ustride] = si;
      u2[(int64_t)i * ustride] = ti;
      y[(int64_t)i * ystride] = bi;
      bi = bnext - mlt * bi;
      double nd = an - mlt * si, ns = bn - mlt * ti;
      di = nd;
      si = ns;
      ti = 0.0;
    } else {
      double mlt = di / ci;
      u0[(int64_t)i * ustride] = ci;
      u1[(int64_t)i * ustride] = an;
      u2[(int64_t)i * ustride] = bn;
      y[(int64_t)i * ystride] = bnext;
      bi = bi - mlt * bnext;
      double nd = si - mlt * an, ns = ti - mlt * bn;
      di = nd;
      si = ns;
      ti = 0.0;
    }
  }
  if (fabs(di) < tiny) di = di < 0.0 ? -tiny : tiny;
  u0[(int64_t)(n - 1) * ustride] = di;
  y[(int64_t)(n - 1) * ystride] = bi;
  // back substitution
  for (int i = n - 1; i >= 0; --i) {
    double s = y[(int64_t)i * ystride];
    if (i + 1 < n) s -= u1[(int64_t)i * ustride] * y[(int64_t)(i + 1) * ystride];
    if (i + 2 < n) s -= u2[(int64_t)i * ustride] * y[(int64_t)(i + 2) * ystride];
    double piv = u0[(int64_t)i * ustride];
    if (fabs(piv) < tiny) piv = piv < 0.0 ? -tiny : tiny;
    y[(int64_t)i * ystride] = s / piv;
  }
}

// One step of the elimination of T - lambda with partial pivoting, rows exchanged
// when sw: the multiplier is at most 1, so the top bit of its exponent is free, and
// there the exchange is kept (in the last bit of its fraction the multiplier lost that
// bit: vectors of a 4096-row chain 25 times further off).
__device__ __forceinline__ double multiplier_of(double num, double piv, double rcp) {
  return fabs(piv) < 0x1p-1000 ? num / piv : num * rcp;  // the reciprocal of a denormal pivot overflows
}
__device__ __forceinline__ double with_exchange(double m, bool sw) {
  return __hiloint2double(__double2hiint(m) | (sw ? 0x40000000 : 0), __double2loint(m));
}
__device__ __forceinline__ bool exchanged(double f) { return (__double2hiint(f) & 0x40000000) != 0; }
__device__ __forceinline__ double multiplier(double f) {
  return __hiloint2double(__double2hiint(f) & ~0x40000000, __double2loint(f));
}

// Inverse iteration for one vector per thread, the arrays interleaved (entry i at
// [i st], so that the threads of a CTA walk the same rows in lockstep and their
// accesses coalesce; loads run PF rows ahead).  T - lambda is factored once, with
// partial pivoting: u0 = 1 / pivot (clamped to +-tiny), u1 the next entry of the row
// and ml the multiplier with the exchange of the rows; the third entry of an exchanged
// row is e[i + 1].  il_factor takes the start vector
// through the elimination as it goes, il_forward any later one.  A chain per row:
// one division in the factorisation, two sums in a solve.  T is in shared memory (in
// global memory no load of it could pass the stores), and a CTA is one warp, so that
// 3072 vectors are spread over 96 SMs.  Factored anew in each of the three
// iterations by CTAs of 128: 2.13 ms at bond dimension 3072 (n <= 1471), now 1.03.
constexpr int PF = 8;
__device__ __forceinline__ double clamped_rcp(double piv, double tiny) {
  return 1.0 / (fabs(piv) < tiny ? (piv < 0.0 ? -tiny : tiny) : piv);
}
template <class Start>
__device__ void il_factor(const double* d, const double* e, int n, double lambda, double tiny, Start start, double* y,
                          double* u0, double* u1, double* ml, int64_t st) {
  double di = d[0] - lambda, si = n > 1 ? e[0] : 0.0, bi = start(0);
#pragma unroll 4
  for (int i = 0; i + 1 < n; ++i) {
    const double ci = e[i], an = d[i + 1] - lambda, bn = i + 2 < n ? e[i + 1] : 0.0, bnext = start(i + 1);
    const bool sw = fabs(di) < fabs(ci);
    if (!sw && di == 0.0) di = tiny;
    const double piv = sw ? ci : di, r = 1.0 / piv;
    const double m = multiplier_of(sw ? di : ci, piv, r);
    u0[i * st] = fabs(piv) < tiny ? clamped_rcp(piv, tiny) : r;
    u1[i * st] = sw ? an : si;
    ml[i * st] = with_exchange(m, sw);
    y[i * st] = sw ? bnext : bi;
    bi = sw ? bi - m * bnext : bnext - m * bi;
    di = sw ? si - m * an : an - m * si;
    si = sw ? -m * bn : bn;
  }
  u0[(n - 1) * st] = clamped_rcp(di, tiny);
  y[(n - 1) * st] = bi;
}
// the elimination applied to y * scale (the iterate before, normalised as it is read)
__device__ void il_forward(int n, double scale, double* y, const double* ml, int64_t st) {
  double bi = y[0] * scale;
  double cb[PF], cm[PF], nb[PF], nm[PF];
  auto load = [&](int i0, double (&b)[PF], double (&m)[PF]) {
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      const bool in = i0 + k + 1 < n;
      b[k] = in ? y[(i0 + k + 1) * st] : 0.0;
      m[k] = in ? ml[(i0 + k) * st] : 0.0;
    }
  };
  load(0, cb, cm);
  for (int i0 = 0; i0 + 1 < n; i0 += PF) {
    load(i0 + PF, nb, nm);
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      if (i0 + k + 1 < n) {
        const double bnext = cb[k] * scale, m = multiplier(cm[k]);
        const bool sw = exchanged(cm[k]);
        y[(i0 + k) * st] = sw ? bnext : bi;
        bi = sw ? bi - m * bnext : bnext - m * bi;
      }
    }
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      cb[k] = nb[k];
      cm[k] = nm[k];
    }
  }
  y[(n - 1) * st] = bi;
}
// back substitution; returns the squared norm of the solution
__device__ double il_back(const double* e, int n, double* y, const double* u0, const double* u1, const double* ml,
                          int64_t st) {
  double x1 = 0.0, x2 = 0.0, ss = 0.0;  // x1, x2: y[i + 1], y[i + 2] as solved
  double cy[PF], c0[PF], c1[PF], c2[PF], ny[PF], n0[PF], n1[PF], n2[PF];
  auto load = [&](int b0, double (&vy)[PF], double (&v0)[PF], double (&v1)[PF], double (&v2)[PF]) {
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      const int i = b0 - k;
      vy[k] = i >= 0 ? y[i * st] : 0.0;
      v0[k] = i >= 0 ? u0[i * st] : 0.0;
      v1[k] = i >= 0 && i + 1 < n ? u1[i * st] : 0.0;
      v2[k] = i >= 0 && i + 2 < n ? ml[i * st] : 0.0;
    }
  };
  load(n - 1, cy, c0, c1, c2);
  for (int b0 = n - 1; b0 >= 0; b0 -= PF) {
    load(b0 - PF, ny, n0, n1, n2);
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      const int i = b0 - k;
      if (i >= 0) {
        const double e1 = exchanged(c2[k]) ? e[i + 1] : 0.0;
        const double xi = fma(-e1, x2, fma(-c1[k], x1, cy[k])) * c0[k];
        y[i * st] = xi;
        ss = fma(xi, xi, ss);
        x2 = x1;
        x1 = xi;
      }
    }
#pragma unroll
    for (int k = 0; k < PF; ++k) {
      cy[k] = ny[k];
      c0[k] = n0[k];
      c1[k] = n1[k];
      c2[k] = n2[k];
    }
  }
  return ss;
}

// U holds the three factor rows back to back (3 n doubles)
__device__ void tri_solve(const double* d, const double* e, int n, double lambda, double tiny, double* y,
                          double* U, int ystride) {
  tri_solve(d, e, n, lambda, tiny, y, U, U + n, U + 2 * n, ystride, 1);
}

__device__ __forceinline__ double hash_unit(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * 0x1.0p-53 * 2.0 - 1.0;
}

// ---------------------------------------------------------------------------
// Eigenvectors of the sectors with n <= SN, one CTA each.
//
// (a) Inverse iteration, one thread per vector: T - lambda I is factored once
//     (one reciprocal per step; the row exchange is kept in the last bit of the
//     multiplier, which the factorisation itself uses too), the INV_ITERS solves
//     then are substitutions only.  Up to 128 rows that bit was seen to move a
//     vector by 2e-14 at most, and a U(1) sweep's single Gram-Schmidt pass can
//     carry any change of a last bit here to 5e-9 in <Sz>, so it stays.
// (b) Gram-Schmidt inside clusters, right-looking and twice: once vector j is
//     final, every warp takes it out of its share of the later members, so a
//     vector costs one barrier.  A vector that the first pass has left less than
//     half of had collapsed onto earlier ones: it is iterated once more from its
//     remainder and projected again.
// (c) Back-transformation z = H_0 H_1 ... H_{n-3} y, four vectors at a time in a
//     warp's registers, without barriers; then the gauge.
// All three are chains of latencies.  Measured against a factorisation per solve,
// Gram-Schmidt vector by vector with eight barriers each and two barriers per
// reflector: at bond dimension 75 (n <= 36) 108 -> 52 us, at 512 (n <= 75) 282 ->
// 116 us.

// Solve with the factors of (T - lambda I): y = the solution for y * scale;
// returns its squared norm.  Entry i of the factors is at [i * st].
__device__ __forceinline__ double small_solve(int n, double scale, double* y, const double* u0, const double* u1,
                                              const double* u2, const double* ml, int st) {
  double bi = y[0] * scale;
#pragma unroll 4
  for (int i = 0; i + 1 < n; ++i) {
    const double bn = y[i + 1] * scale, m = ml[i * st];
    const bool sw = __double2loint(m) & 1;
    const double top = sw ? bn : bi, low = sw ? bi : bn;
    y[i] = top;
    bi = fma(-m, top, low);
  }
  double x1 = 0.0, x2 = 0.0, ss = 0.0;
  double s = bi;
#pragma unroll 4
  for (int i = n - 1; i >= 0; --i) {
    if (i < n - 1) s = y[i] - u1[i * st] * x1 - u2[i * st] * x2;
    const double xi = s * u0[i * st];
    y[i] = xi;
    ss = fma(xi, xi, ss);
    x2 = x1;
    x1 = xi;
  }
  return ss;
}

__host__ __device__ constexpr int64_t small_vec_smem(int n, int nvec) { return 4 * (int64_t)n + (int64_t)nvec * (n | 1); }

__global__ void __launch_bounds__(TT, 1)
eigvecs_small(const EigDev* __restrict__ probs, const double* G, const double* Tg, const double* W, double* Zg,
              double* work, const double* Amat, int64_t cap) {
  extern __shared__ double zsm[];
  __shared__ double red[33];
  __shared__ double coef[SN];
  __shared__ unsigned begins[SB];  // bit j: vector j begins a cluster
  // the GPU-wide kernel that may follow reads nothing of this one's
  asm volatile("griddepcontrol.launch_dependents;");
  const EigDev P = probs[blockIdx.x];
  const int n = P.n, cnt = P.nvec;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  if (n <= 0 || cnt <= 0) return;
  double* Zout = Zg + P.g_off;  // n x cnt, leading dimension n
  if (P.flags & TT_EIG_ROW_1X2) {
    if (tid == 0) {
      double a = Amat[P.a_off], b = Amat[P.a_off + 1];
      double dd = sqrt(a * a + b * b), z0, z1;
      if (dd != 0.0) {
        double inv = 1.0 / dd;
        z0 = a * inv;
        z1 = b * inv;
      } else {
        z0 = z1 = 1.0 / sqrt(2.0);
      }
      Zout[0] = z0;
      Zout[1] = z1;
      if (cnt > 1) {
        Zout[2] = -z1;
        Zout[3] = z0;
      }
    }
    return;
  }
  const double* tau = Tg + 3 * P.w_off + 2 * n;
  const double* Gp = G + P.g_off;
  const int ld = n | 1;  // odd: the threads' vectors lie on different banks
  double* d = zsm;
  double* e = d + n;
  double* lam = e + n;    // descending
  double* Z = lam + 2 * n;  // [cnt][ld]
  // the factors, per vector: in shared memory when they fit, else interleaved
  // in the work area and (u2) in the output
  const bool fits = small_vec_smem(n, cnt) + 4 * (int64_t)cnt * ld <= cap;
  double* u0 = fits ? Z + (int64_t)cnt * ld : work + 3 * P.g_off;
  double* u1 = u0 + (int64_t)cnt * (fits ? ld : n);
  double* ml = u1 + (int64_t)cnt * (fits ? ld : n);
  double* u2 = fits ? ml + (int64_t)cnt * ld : Zout;
  const int st = fits ? 1 : cnt, sv = fits ? ld : 1;  // from entry to entry, from vector to vector
  for (int i = tid; i < n; i += blockDim.x) {
    d[i] = Tg[3 * P.w_off + i];
    e[i] = i + 1 < n ? Tg[3 * P.w_off + n + i] : 0.0;
    if (i < cnt) lam[i] = W[P.w_off + i];
  }
  __syncthreads();
  double loc = 0.0;
  for (int i = tid; i < n; i += blockDim.x) loc = fmax(loc, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + fabs(e[i]));
  double tnorm = block_reduce(loc, red, true);
  if (tnorm > 0.0 && isfinite(tnorm)) {  // a norm in [1/2, 1), so that no solution overflows when it is squared
    int ex;
    frexp(tnorm, &ex);
    tnorm = ldexp(tnorm, -ex);
    for (int i = tid; i < n; i += blockDim.x) {
      d[i] = ldexp(d[i], -ex);
      e[i] = ldexp(e[i], -ex);
      if (i < cnt) lam[i] = ldexp(lam[i], -ex);
    }
    __syncthreads();
  }
  // pivot floor; a zero T takes 1 so that b / tiny cannot overflow
  const double tiny = tnorm > 0.0 ? DBL_EPSILON * tnorm : 1.0;
  const double ortol = 1e-3 * tnorm;
  auto clamped = [&](double p) { return fabs(p) < tiny ? (p < 0.0 ? -tiny : tiny) : p; };
  auto solve = [&](int j, double scale) {
    return small_solve(n, scale, Z + (int64_t)ld * j, u0 + (int64_t)sv * j, u1 + (int64_t)sv * j, u2 + (int64_t)sv * j,
                       ml + (int64_t)sv * j, st);
  };
  if (tid < SB * 32) {
    const bool first = tid < cnt && (tid == 0 || lam[tid - 1] - lam[tid] > ortol);
    const unsigned m = __ballot_sync(0xffffffffu, first);
    if (lane == 0) begins[warp] = m;
  }
  // (a)
  if (tid < cnt) {
    const int j = tid;
    double* y = Z + (int64_t)ld * j;
    double* f0 = u0 + (int64_t)sv * j;
    double* f1 = u1 + (int64_t)sv * j;
    double* f2 = u2 + (int64_t)sv * j;
    double* fm = ml + (int64_t)sv * j;
    const double lj = lam[j];
    double di = d[0] - lj, si = e[0];
    for (int i = 0; i + 1 < n; ++i) {
      const double ci = e[i], an = d[i + 1] - lj, bn = e[i + 1];
      const bool sw = fabs(di) < fabs(ci);
      if (!sw && di == 0.0) di = tiny;
      const double piv = sw ? ci : di, r = 1.0 / piv;
      double m = (sw ? di : ci) * r;
      m = __hiloint2double(__double2hiint(m), (__double2loint(m) & ~1) | (sw ? 1 : 0));
      f0[i * st] = fabs(piv) < tiny ? 1.0 / clamped(piv) : r;
      f1[i * st] = sw ? an : si;
      f2[i * st] = sw ? bn : 0.0;
      fm[i * st] = m;
      di = sw ? si - m * an : an - m * si;
      si = sw ? -m * bn : bn;
    }
    f0[(n - 1) * st] = 1.0 / clamped(di);
    f1[(n - 1) * st] = f2[(n - 1) * st] = 0.0;
    for (int i = 0; i < n; ++i) y[i] = hash_unit(((uint64_t)P.g_off << 20) ^ ((uint64_t)j << 32) ^ (uint64_t)i);
    double scale = 1.0;
    for (int it = 0; it < INV_ITERS; ++it) scale = 1.0 / sqrt(solve(j, scale));
    for (int i = 0; i < n; ++i) y[i] *= scale;
  }
  __syncthreads();
  // (b)
  auto next_begin = [&](int j) {  // the first vector after j that begins a cluster (cnt: none)
    for (int w = (j + 1) >> 5; w < SB; ++w) {
      const unsigned m = begins[w] & (w == (j + 1) >> 5 ? 0xffffffffu << ((j + 1) & 31) : 0xffffffffu);
      if (m) return 32 * w + __ffs(m) - 1;
    }
    return cnt;
  };
  auto dot = [&](const double* a, const double* b) {
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += a[i] * b[i];
    return warp_sum(s);
  };
  for (int pass = 0; pass < 2; ++pass) {
    for (int c0 = 0; c0 < cnt;) {
      const int c1 = next_begin(c0);
      for (int j = c0; j < c1 && c1 - c0 > 1; ++j) {
        double* y = Z + (int64_t)ld * j;
        double nn = dot(y, y);  // every warp alike
        if (pass == 0 && j > c0 && !(nn > 0.25)) {
          for (int tries = 0; tries < 5; ++tries) {
            __syncthreads();
            if (tid == 0) {
              const double nrm = sqrt(nn);
              if (!(nrm > 0.0))
                for (int i = 0; i < n; ++i) y[i] = hash_unit((uint64_t)(j * 7919 + i + tries));
              solve(j, nrm > 0.0 ? 1.0 / nrm : 1.0);
            }
            __syncthreads();
            for (int r = 0; r < 2; ++r) {
              for (int k = c0 + warp; k < j; k += nw) {
                const double* z = Z + (int64_t)ld * k;
                const double q = dot(z, y) / dot(z, z);
                if (lane == 0) coef[k] = q;
              }
              __syncthreads();
              if (tid < n) {
                double s = y[tid];
                for (int k = c0; k < j; ++k) s -= coef[k] * Z[(int64_t)ld * k + tid];
                y[tid] = s;
              }
              __syncthreads();
            }
            nn = dot(y, y);
            if (nn > 0.25) break;
          }
          __syncthreads();
          const double inv = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
          if (tid < n) y[tid] *= inv;
          __syncthreads();
          nn = dot(y, y);
        }
        if (j + 1 == c1) continue;
        const double inv = nn > 0.0 ? 1.0 / nn : 0.0;
        for (int k = j + 1 + warp; k < c1; k += nw) {
          double* z = Z + (int64_t)ld * k;
          const double q = dot(y, z) * inv;
          for (int i = lane; i < n; i += 32) z[i] -= q * y[i];
        }
        __syncthreads();
      }
      c0 = c1;
    }
  }
  __syncthreads();
  // (c)
  constexpr int VB = 4;
  for (int t0 = VB * warp; t0 < cnt; t0 += VB * nw) {
    double y[VB][SB];
#pragma unroll
    for (int u = 0; u < VB; ++u) {
      double s = 0.0;
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int r = lane + 32 * b;
        y[u][b] = t0 + u < cnt && r < n ? Z[(int64_t)ld * (t0 + u) + r] : 0.0;
        s += y[u][b] * y[u][b];
      }
      s = warp_sum(s);
      const double inv = s > 0.0 ? 1.0 / sqrt(s) : 0.0;
#pragma unroll
      for (int b = 0; b < SB; ++b) y[u][b] *= inv;
    }
    double vnx[SB], tnx = 0.0;  // the next reflector, loaded one step ahead
    auto load = [&](int k) {
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int r = lane + 32 * b;
        vnx[b] = k >= 0 && r >= k + 1 && r < n ? (r == k + 1 ? 1.0 : Gp[r + n * k]) : 0.0;
      }
      tnx = k >= 0 ? tau[k] : 0.0;
    };
    load(n - 3);
    for (int k = n - 3; k >= 0; --k) {
      double v[SB];
#pragma unroll
      for (int b = 0; b < SB; ++b) v[b] = vnx[b];
      const double tk = tnx;
      load(k - 1);
      double s[VB];
#pragma unroll
      for (int u = 0; u < VB; ++u) {
        s[u] = 0.0;
#pragma unroll
        for (int b = 0; b < SB; ++b) s[u] = fma(v[b], y[u][b], s[u]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < VB; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
#pragma unroll
      for (int u = 0; u < VB; ++u)
#pragma unroll
        for (int b = 0; b < SB; ++b) y[u][b] = fma(-tk * s[u], v[b], y[u][b]);
    }
    // deterministic gauge: the largest-magnitude entry (first on ties) is positive
#pragma unroll
    for (int u = 0; u < VB; ++u) {
      double best = -1.0;
      int bi = n;
      bool neg = false;
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int r = lane + 32 * b;
        const double m = fabs(y[u][b]);
        if (r < n && m > best) {
          best = m;
          bi = r;
          neg = y[u][b] < 0.0;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        const bool on = __shfl_xor_sync(0xffffffffu, (int)neg, o);
        if (ob > best || (ob == best && oi < bi)) {
          best = ob;
          bi = oi;
          neg = on;
        }
      }
      if (t0 + u < cnt)
#pragma unroll
        for (int b = 0; b < SB; ++b) {
          const int r = lane + 32 * b;
          if (r < n) Zout[r + (int64_t)n * (t0 + u)] = neg ? -y[u][b] : y[u][b];
        }
    }
  }
}

// ---------------------------------------------------------------------------
// Sectors with n > SN: one thread-block cluster (CL CTAs, distributed shared
// memory) per sector, so a large density matrix is reduced by CL SMs at once
// instead of one SM streaming it from L2.
//
// Phase 1: Householder tridiagonalisation with the rank-2 updates of up to nb
// reflectors pending (Golub & Van Loan, "Matrix Computations", 4th ed., sec.
// 8.3.1).  CTA q owns the columns c % CL == q, whole (both triangles), in shared
// memory when they fit, else in a scratch of its own in L2; every CTA holds the
// pending v and w on all rows.  So CTA q forms (A0 v)_c of its own columns c
// without help, A0 the matrix as of the last flush, and one exchange per column
// is enough: to every CTA go, for every own column c, (A0 v)_c and -- the matrix
// is symmetric -- the entry A0[k+1, c] of the next column, and the CTA's shares of
// v^T A0 v and of the pending V^T v and W^T v.  After the cluster barrier every
// CTA forms for itself, on all rows and from the same data,
//   p = A0 v - V (W^T v) - W (V^T v),  w = tau p - (tau^2 / 2)(v^T p) v,
//   x = A0[:, k+1] - V W[k+1]^T - W V[k+1]^T   (this reflector included),
// and from x the next reflector: one block-wide reduction (sigma) and one
// barrier (v is complete) before the next products.  When nb reflectors are
// pending, the products' pass over the own columns applies them on the way.
// What a CTA pushes for column k + 1 may arrive while another still reads what it
// got for column k, so the arrays pushed to are double (by parity).
//
// Phase 2: CTA r owns eigenvectors [r q, r q + q), q = ceil(nvec / CL).
// Inverse iteration runs one thread per vector.  Gram-Schmidt (twice, inside
// the clusters of close eigenvalues as in the one-CTA kernel) takes vectors
// in order: each CTA projects the current vector y on its own earlier cluster
// members and publishes the partial sum of projections; after a cluster
// barrier every CTA subtracts all partial sums in CTA order.  Every CTA thus
// holds the same iterate, decides collapse/retry identically, and one barrier
// per projection round suffices (partial sums alternate between two buffers).
// The back-transformation needs no communication: every CTA applies all
// reflectors to its own vectors, staged a few at a time in shared memory.
// Every loop bound here is the same in all CTAs of a cluster, so every CTA
// reaches every cluster barrier.
namespace cgx = cooperative_groups;

constexpr int CL_STAGE = 4;  // reflectors staged per round of the back-transformation
constexpr int CL_MAX = 16;   // largest cluster the kernels are launched with
constexpr int NWARP = TT / 32;
constexpr int NB_MAX = 16;   // pending reflectors of the cluster reduction, at most
constexpr int CR_THREADS = 256;  // its threads per CTA
constexpr int CR_STAGE = 64;     // columns between its layouts (a multiple of CL_MAX)
struct VecTaskB {
  int32_t prob, j0;  // problem (index into the problem array) and first eigenvalue
};

__device__ __host__ __forceinline__ int first_owned(int from, int rank, int CL) {
  // smallest l with rank + CL * l >= from
  return from <= rank ? 0 : (from - rank + CL - 1) / CL;
}

constexpr int PNB_MAX = 32;      // widest panel of the blocked reduction

// doubles of dynamic shared memory of the blocked cluster reduction
__host__ __device__ inline int64_t blocked_smem(int n, int nb, int CL) {
  const int64_t nloc = (n + CL - 1) / CL;
  return 2 * (int64_t)nb * nloc        // V, W of the panel on the own rows
         + 2 * nloc                    // the own rows of the current and the next column
         + (int64_t)CL * nloc          // the pushed column, then v, owner-major
         + (int64_t)CL * nloc          // this CTA's row sums of A22 v, owner-major
         + (int64_t)CL * nloc          // pushed row sums of A22 v on the own rows, per sender
         + (int64_t)NWARP * nloc       // per-warp column dots
         + CL_MAX * 2 * (int64_t)nb    // pushed V^T v, W^T v partials
         + CL_MAX                      // pushed v^T A22 v partials
         + CL_MAX * (int64_t)nb        // pushed row sums on the panel's rows
         + nb                          // pushed column dots of the panel's rows
         + 2 * (int64_t)nb * nb        // V, W on the panel's rows
         + 2 * (int64_t)nb;            // V^T v, W^T v
}

// Shared memory of the cluster reduction, in doubles, for the n rows and columns
// that are left: nb pending reflectors (v, w) on all rows and (w, v) on the own
// columns, the current v, the pushed pairs (twice), the pushed partial sums, and the
// own columns when they are resident.
constexpr int CLR_MISC = 2 * CL_MAX * 2 * NB_MAX + 2 * CL_MAX * NWARP + NWARP * 2 * NB_MAX;
struct ClusterLayout {
  int nb;           // pending reflectors (0: does not fit)
  bool resident;    // own columns in shared memory
  int64_t doubles;  // in all
};
__host__ __device__ inline int cl_ld(int n) { return (n + 2) & ~1; }  // rows of a column: even, at least one of padding
__host__ __device__ inline ClusterLayout cluster_layout(int n, int CL, int64_t cap) {
  const int64_t ld = cl_ld(n), nloc = (n + CL - 1) / CL;
  for (const bool resident : {true, false}) {
    const int64_t fixed = CLR_MISC + 5 * ld + (resident ? nloc * ld : 0);
    int64_t nb = fixed < cap ? (cap - fixed) / (2 * (ld + nloc)) : 0;
    if (nb > NB_MAX) nb = NB_MAX;
    // resident columns pay when a few reflectors still fit beside them (n = 470, 6 and
    // in L2 16 pending: 1.88 and 2.04 ms; from 2 on 540 would take 2.29 ms for 2.43, 700 as
    // long)
    if (nb < (resident ? 6 : 1)) continue;
    return ClusterLayout{(int)nb, resident, fixed + nb * 2 * (ld + nloc)};
  }
  return ClusterLayout{0, false, 0};
}

// D += A B for one m8n8k4 FP64 tile (DMMA): A 8x4 row fragment (lane L holds
// A[L/4][L%4]), B 4x8 column fragment (B[L%4][L/4]), D 8x8 (D[L/4][2(L%4)+e])
__device__ __forceinline__ void dmma_tr(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// The pending reflectors applied to the own columns l >= lf, rows from rs (even) on:
// A -= V W^T + W V^T on the FP64 tensor path, a warp per 32 rows x 16 columns as the
// transposed product (a lane's pair of results is two rows of a column: 16-byte
// accesses).  vw: (v, w)
// on all rows; wv: (w, v) on the own columns.
template <int NW>
__device__ __noinline__ void cluster_flush(double* cols, int ld, int rend, int lf, int lown, int rs, int np,
                                           const double2* vw, int ldv, const double2* wv, int ldw, int warp, int lane) {
  const int g = lane >> 2, t4 = lane & 3;
  const int ncb = (lown - lf + 15) >> 4, nrt = (rend - rs + 31) >> 5;
  const double* va = reinterpret_cast<const double*>(vw) + (t4 & 1);
  const double* vb = reinterpret_cast<const double*>(wv) + (t4 & 1);
  // columns and rows past the end read a valid element, which is not stored
  auto tile = [&](int task, bool store, double (&acc)[2][4][2]) {
    const int r0 = rs + 32 * (task / ncb) + 2 * t4, lb = lf + 16 * (task % ncb) + g;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int l = lb + 8 * b;
      double* col = cols + (int64_t)min(l, lown - 1) * ld;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + 8 * i;
        if (!store) {
          const double2 x = *reinterpret_cast<const double2*>(col + min(r, rend - 2));
          acc[b][i][0] = x.x;
          acc[b][i][1] = x.y;
        } else if (r < rend && l < lown) {
          *reinterpret_cast<double2*>(col + r) = make_double2(acc[b][i][0], acc[b][i][1]);
        }
      }
    }
  };
  const int tasks = ncb * nrt;
  auto update = [&](int task, double (&acc)[2][4][2]) {
    const int r0 = rs + 32 * (task / ncb) + g, lb = lf + 16 * (task % ncb) + g;
    for (int t0 = 0; t0 < np; t0 += 2) {
      const int t = min(t0 + (t4 >> 1), np - 1);
      const bool in = t0 + (t4 >> 1) < np;
      double af[2], bf[4];
#pragma unroll
      for (int b = 0; b < 2; ++b) af[b] = in ? -vb[2 * (t * ldw + min(lb + 8 * b, lown - 1))] : 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) bf[i] = in ? va[2 * ((int64_t)t * ldv + min(r0 + 8 * i, rend - 1))] : 0.0;
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) dmma_tr(acc[b][i], af[b], bf[i]);
    }
    tile(task, true, acc);
  };
  // two tiles in turn, so that one is in flight while the other is updated
  double t0[2][4][2], t1[2][4][2];
  int task = warp;
  if (task < tasks) tile(task, false, t0);
  if (task + NW < tasks) tile(task + NW, false, t1);
  for (; task < tasks; task += 2 * NW) {
    update(task, t0);
    if (task + 2 * NW < tasks) tile(task + 2 * NW, false, t0);
    if (task + NW < tasks) update(task + NW, t1);
    if (task + 3 * NW < tasks) tile(task + 3 * NW, false, t1);
  }
}

// One pass over the own columns l >= lf of a CTA: A0[:, c] . v over the rows from
// rs on (even), pushed with A0[row, c] to every CTA; returns this warp's share of
// v^T A0 v.  A warp takes two columns at a time, 64 U rows of each per step.
template <int NW, int U>
__device__ __forceinline__ double cluster_pass(const double* cols, int ld, int rend, int lf, int lown,
                                               int rank, int CL, int rs, int row, const double* vcur, double2* push,
                                               int warp, int lane) {
  cgx::cluster_group cluster = cgx::this_cluster();
  double share = 0.0;
  auto load = [&](int l, int rc, double2 (&a)[2][U]) {
    const double* q0 = cols + (int64_t)l * ld + rc + 2 * lane;
    const double* q1 = l + 1 < lown ? q0 + ld : q0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = rc + 2 * lane + 64 * u < rend;
      a[0][u] = in ? *reinterpret_cast<const double2*>(q0 + 64 * u) : make_double2(0.0, 0.0);
      a[1][u] = in ? *reinterpret_cast<const double2*>(q1 + 64 * u) : make_double2(0.0, 0.0);
    }
  };
  auto emit = [&](int l, double s) {
    const int c = rank + CL * l;
    const double2 out = make_double2(s, cols[(int64_t)l * ld + row]);
    if (lane < CL) *cluster.map_shared_rank(push + c, lane) = out;
    share += s * vcur[c];
  };
  double s0 = 0.0, s1 = 0.0;
  auto use = [&](int l, int rc, const double2 (&a)[2][U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = rc + 2 * lane + 64 * u;
      const double2 v = r < rend ? *reinterpret_cast<const double2*>(vcur + r) : make_double2(0.0, 0.0);
      s0 = fma(a[0][u].x, v.x, fma(a[0][u].y, v.y, s0));
      s1 = fma(a[1][u].x, v.x, fma(a[1][u].y, v.y, s1));
    }
    if (rc + 64 * U < rend) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    }
    emit(l, s0);
    if (l + 1 < lown) emit(l + 1, s1);
    s0 = s1 = 0.0;
  };
  // two steps in turn, so that one is in flight while the other is used
  int l0 = lf + 2 * warp, r0 = rs, l1 = l0, r1 = r0;
  auto after = [&](int l, int rc, int& ln, int& rn) {  // the step after (l, rc)
    ln = l;
    rn = rc + 64 * U;
    if (rn >= rend) {
      ln = l + 2 * NW;
      rn = rs;
    }
  };
  double2 b0[2][U], b1[2][U];
  if (l0 < lown) load(l0, r0, b0);
  after(l0, r0, l1, r1);
  if (l1 < lown) load(l1, r1, b1);
  while (l0 < lown) {
    use(l0, r0, b0);
    after(l1, r1, l0, r0);
    if (l0 < lown) load(l0, r0, b0);
    if (l1 >= lown) break;
    use(l1, r1, b1);
    after(l0, r0, l1, r1);
    if (l1 < lown) load(l1, r1, b1);
  }
  return share;
}

// RPT: rows of a thread, at least n / CR_THREADS.  256 threads: what every warp
// does for itself costs half of what it would with 512, and 255 registers a thread
// hold two steps of loads (eight columns' worth spilled, and a spill goes to L2
// beside 220 KB of shared memory: 10 ms more at n = 1471).
//
// Measured with clocks in the kernel, n = 1471 (17 ms in all): the pass over the
// own columns 8 (their reads from L2 while they do not fit), flushes 3.7, rows 2.1,
// cluster barrier 1.4, the reflector 1.3.  Against the blocked
// reduction with two barriers per column, panels of 32 and the row sums of a lower
// triangle exchanged: block SVD's reduction at bond dimension 3072 (n <= 1471)
// 22.3 -> 17.2 ms, at 512 (n <= 245, columns resident) 2.33 -> 0.79 ms.
template <int RPT>
__global__ void __launch_bounds__(CR_THREADS, 1)
tridiag_eigvals_cluster(const EigDev* __restrict__ probs, double* G, double* Tg, double* scratch,
                        int64_t cap) {
  extern __shared__ double sm[];
  constexpr int NT = CR_THREADS, NW = NT / 32, U = 4;
  __shared__ double red[NW], s_x[2];
  cgx::cluster_group cluster = cgx::this_cluster();
  const int CL = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const EigDev P = probs[blockIdx.x / CL];
  const int n = P.n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* Gp = G + P.g_off;
  double* dg = Tg + 3 * P.w_off;
  double* eg = dg + n;
  double* tg = eg + n;
  const int rend = cl_ld(n);  // end of the (zero-padded) rows
  const int nloc = (n + CL - 1) / CL, lg = __ffs(CL) - 1;  // CL is a power of two
  const int lown = first_owned(n, rank, CL);  // own columns c = rank + CL l, l < lown
  double* gcols = scratch + P.s_off + (int64_t)rank * nloc * rend;  // the own columns in L2, [lown][rend]
  // Shared memory, laid out for the rows and columns from o on (a multiple of CL)
  // and again every CR_STAGE columns: the fewer are left, the more reflectors may
  // be pending, until the own columns fit as well.  All pointers take the absolute
  // row r or own column l.
  int o = 0, nb = 0, ldv = 0, ldw = 0, ldc = rend;
  bool resident = false;
  double2 *vw = nullptr, *push = nullptr, *part = nullptr, *ab = nullptr, *wv = nullptr;
  double *vcur = nullptr, *vav = nullptr, *cols = nullptr;
  auto lay_out = [&](int from) {
    const ClusterLayout L = cluster_layout(n - from, CL, cap);
    o = from;
    nb = L.nb;
    resident = L.resident;
    ldv = rend - o;
    ldw = nloc - o / CL;
    vw = reinterpret_cast<double2*>(sm) - o;                     // [nb][ldv]: (v, w)
    vcur = sm + (int64_t)nb * 2 * ldv - o;                       // [ldv]
    push = reinterpret_cast<double2*>(vcur + o + ldv) - o;       // [2][ldv]: (A0 v, A0[:, k + 1])
    part = push + o + 2 * ldv;                                   // [2][CL_MAX][NB_MAX]: shares of (W^T v, V^T v)
    vav = reinterpret_cast<double*>(part + 2 * CL_MAX * NB_MAX);  // [2][CL_MAX][NW]: shares of v^T A0 v
    ab = reinterpret_cast<double2*>(vav + 2 * CL_MAX * NWARP) + warp * NB_MAX;  // this warp's (W^T v, V^T v)
    wv = reinterpret_cast<double2*>(reinterpret_cast<double*>(part) + CLR_MISC) - o / CL;  // [nb][ldw]: (w, v) on the own columns
    ldc = resident ? ldv : rend;
    cols = resident ? reinterpret_cast<double*>(wv + o / CL + nb * ldw) - (int64_t)(o / CL) * ldc - o : gcols;
  };
  lay_out(0);
  for (int l = warp; l < lown; l += NW)
    for (int r = lane; r < rend; r += 32)
      cols[(int64_t)l * ldc + r] = r < n ? Gp[r + (int64_t)n * (rank + CL * l)] : 0.0;
  auto zero_padding = [&]() {
    for (int i = tid; i < nb * (rend - n); i += NT)
      vw[(int64_t)(i / (rend - n)) * ldv + n + i % (rend - n)] = make_double2(0.0, 0.0);
    if (tid < rend - n) vcur[n + tid] = 0.0;
  };
  zero_padding();
  double x[RPT];  // the next column on the rows tid + TT i
#pragma unroll
  for (int i = 0; i < RPT; ++i) x[i] = tid + NT * i < n ? Gp[tid + NT * i] : 0.0;
  __threadfence_block();
  cluster.sync();  // column 0 is read; its owner overwrites it
  int np = 0, par = 0;
  for (int k = 0; k + 2 < n; ++k) {
    if (!resident && k > 0 && k % CR_STAGE == 0) {  // lay out again (x stays in registers)
      __syncthreads();
      if (np > 0) cluster_flush<NW>(cols, ldc, rend, first_owned(k, rank, CL), lown, k, np, vw, ldv, wv, ldw, warp, lane);
      np = 0;
      cluster.sync();  // nobody reads the old layout any more
      lay_out(k);
      if (resident)
        for (int l = o / CL + warp; l < lown; l += NW)
          for (int r = o + lane; r < rend; r += 32) cols[(int64_t)l * ldc + r] = gcols[(int64_t)l * rend + r];
      zero_padding();
      cluster.sync();  // the new one is ready to be pushed to
    }
    // ---- the reflector of column k (every CTA alike) ----
    double sig = 0.0;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + NT * i;
      if (r >= k + 2 && r < n) sig += x[i] * x[i];
      if (r == k) s_x[0] = x[i];
      if (r == k + 1) s_x[1] = x[i];
    }
    sig = warp_sum(sig);
    if (lane == 0) red[warp] = sig;
    __syncthreads();
    double part_s[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) part_s[w] = red[w];
#pragma unroll
    for (int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
      for (int w = 0; w < o; ++w) part_s[w] += part_s[w + o];
    const double sigma = part_s[0], alpha = s_x[1];
    // beta = -sign(alpha) |(alpha, sigma)|, tau = (beta - alpha) / beta, v = x / (alpha - beta)
    double tau = 0.0, beta = alpha, scale = 0.0;
    if (sigma != 0.0) {
      const double s2 = fma(alpha, alpha, sigma), ri = rsqrt(s2), mu = s2 * ri;
      beta = alpha <= 0.0 ? mu : -mu;
      tau = fma(fabs(alpha), ri, 1.0);
      scale = 1.0 / (alpha - beta);
    }
    const bool owner = rank == k % CL;
    if (owner && tid == 0) {
      dg[k] = s_x[0];
      eg[k] = beta;
      tg[k] = tau;
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + NT * i;
      if (r >= k && r < n) {
        const double v = r == k + 1 ? 1.0 : (r == k ? 0.0 : x[i] * scale);
        vcur[r] = v;
        if (owner && r >= k + 2) Gp[r + (int64_t)n * k] = v;  // kept below the subdiagonal for phase 2
      }
    }
    __syncthreads();
    // ---- the shares of the pending V^T v and W^T v, and A0 v on the own columns ----
    const bool flush = np == nb;
    double2* pushed = push + par * ldv;
    double2* mypart = part + par * CL_MAX * NB_MAX;
    double* myvav = vav + par * CL_MAX * NWARP;
    const int lf = first_owned(k + 1, rank, CL), rs = (k + 1) & ~1;
    if (flush) {
      cluster_flush<NW>(cols, ldc, rend, lf, lown, rs, np, vw, ldv, wv, ldw, warp, lane);
      np = 0;
      __syncthreads();
    }
    for (int t = warp; t < np; t += NW) {
      const double2* p = vw + (int64_t)t * ldv;
      const int seg = (n - k - 1 + CL - 1) / CL, r0 = k + 1 + rank * seg, r1 = min(n, r0 + seg);
      double a = 0.0, b = 0.0;
      for (int r = r0 + lane; r < r1; r += 32) {
        const double2 y = p[r];
        const double v = vcur[r];
        a = fma(y.y, v, a);
        b = fma(y.x, v, b);
      }
      a = warp_sum(a);
      b = warp_sum(b);
      if (lane < CL) *cluster.map_shared_rank(mypart + rank * NB_MAX + t, lane) = make_double2(a, b);
    }
    const double share = cluster_pass<NW, U>(cols, ldc, rend, lf, lown, rank, CL, rs, k + 1, vcur, pushed, warp, lane);
    if (lane < CL) *cluster.map_shared_rank(myvav + rank * NW + warp, lane) = share;
    cluster.sync();
    // ---- w and the next column, on all rows (every CTA alike; the sums by every warp for itself) ----
    const int t = lane & 15, half = lane >> 4;  // two lanes per pending reflector, each every other CTA's share
    double a = 0.0, b = 0.0, s = 0.0;
#pragma unroll
    for (int u = 0; u < CL_MAX / 2; ++u) {
      const int q = 2 * u + half;
      if (t < np && q < CL) {
        const double2 y = mypart[q * NB_MAX + t];
        a += y.x;
        b += y.y;
      }
    }
#pragma unroll
    for (int u = 0; u < CL_MAX * NW / 32; ++u)
      if (lane + 32 * u < CL * NW) s += myvav[lane + 32 * u];
    a += __shfl_xor_sync(0xffffffffu, a, 16);
    b += __shfl_xor_sync(0xffffffffu, b, 16);
    double pc = 0.0;  // V (W^T v) + W (V^T v) at row k + 1
    if (lane < np) {
      const double2 y = vw[(int64_t)lane * ldv + k + 1];
      pc = fma(y.x, a, y.y * b);
      s = fma(-2.0 * a, b, s);
      ab[lane] = make_double2(a, b);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      pc += __shfl_xor_sync(0xffffffffu, pc, o);
    }
    const double K = 0.5 * tau * tau * s;
    const double wk1 = tau * (pushed[k + 1].x - pc) - K;  // w at row k + 1, where v is 1
    __syncwarp();
    double p[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + NT * i;
      const double2 y = r > k && r < n ? pushed[r] : make_double2(0.0, 0.0);
      p[i] = y.x;
      x[i] = y.y;
    }
    for (int u = 0; u < np; ++u) {
      const double2 f = vw[(int64_t)u * ldv + k + 1], q = ab[u];
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = tid + NT * i;
        if (r > k && r < n) {
          const double2 z = vw[(int64_t)u * ldv + r];
          p[i] = fma(-z.x, q.x, fma(-z.y, q.y, p[i]));
          x[i] = fma(-z.x, f.y, fma(-z.y, f.x, x[i]));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + NT * i;
      if (r > k && r < n) {
        const double v = vcur[r];
        const double w = tau * p[i] - K * v;
        x[i] = x[i] - v * wk1 - w;
        vw[(int64_t)np * ldv + r] = make_double2(v, w);
        if ((r & (CL - 1)) == rank) wv[np * ldw + (r >> lg)] = make_double2(w, v);
      }
    }
    ++np;
    par ^= 1;
  }
  // T: the last 2 x 2 block
  __syncthreads();
  if (rank == 0) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + NT * i;
      if (r == n - 2) dg[n - 2] = x[i];
      if (r == n - 1) eg[n - 2] = x[i];
    }
    if (tid == 0) {
      eg[n - 1] = 0.0;
      tg[n - 1] = 0.0;
      tg[n - 2] = 0.0;
    }
  }
  if (rank == (n - 1) % CL && tid == 0) {
    double t = cols[(int64_t)(lown - 1) * ldc + n - 1];
    for (int q = 0; q < np; ++q) {
      const double2 z = vw[(int64_t)q * ldv + n - 1];
      t -= 2.0 * z.x * z.y;
    }
    dg[n - 1] = t;
  }
  cluster.sync();  // the last access of another CTA's shared memory
  // launched alongside tridiag_small: complete only when that is
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The largest sectors: the blocked reduction of LAPACK's dsytrd / dlatrd (Golub & Van
// Loan, ibid., with the panel form of sec. 5.1.7).  The reflectors of a panel of nb
// columns are formed one by one against the matrix as it stood at the start of the
// panel, corrected on the fly by the panel's V and W (A22 v - V W^T v - W V^T v), and
// the trailing matrix receives the rank-2nb update A -= V W^T + W V^T once per panel.
// Only the lower triangle is read or updated, in place.  Index c (row or column)
// belongs to CTA c % CL.  Per column j, two cluster barriers:
//   1. the owners of rows >= j bring column j up to date and push it to every CTA;
//   2. every CTA forms the same reflector from the whole column (same data, same
//      reduction order), keeps v, and pushes its partial V^T v, W^T v;
//   3. every CTA runs A22 v over the lower triangle of its own columns: one warp per
//      block of 64 rows, each lane two rows, columns 16 at a time; an element A[i,c]
//      (i >= c) adds A[i,c] v_i to the dot of column c and, below the diagonal,
//      A[i,c] v_c to row i.  The column dots are summed across the lanes by a butterfly
//      reduce-scatter, the row sums go to the row's owner (a slot per sender), and the
//      CTA's share of v^T A22 v to every CTA;
//   4. every CTA completes p = A22 v on its own rows (own dot + the pushed row sums, in
//      CTA order), w' = tau (p - V W^T v - W V^T v) and w = w' - (tau/2)(w'.v) v; the
//      panel's rows, which every CTA needs, have their sums pushed to every CTA.
// Every CTA sums pushed partials in CTA order, so every decision and scalar is the same
// in every CTA.  The trailing update goes through a global n x 2nb scratch.
//
// The reduction above holds its pending reflectors on all rows in every CTA, so the
// larger the sector the fewer it can hold (6 at n = 1471, 3 at 2048, 1 at 3000) and the
// more often both triangles go through L2; here a CTA holds 8 to 32 on its own rows
// only, and half of the matrix moves.  Measured (this / that, ms): one sector of 1750
// 31.4 / 27.2, 2048 45.3 / 40.5, 2200 46.9 / 55.3, 3000 91.9 / 158, 4096 219 / 573; four
// of 1750 32.5 / 29.5, 1900 37.3 / 40.6, 2048 48.0 / 53.5: the rule is blocked_sectors.
// acc[k] (k < 16) summed over the 32 lanes of the warp, lane L receiving the
// sum of index L % 16: a butterfly sum across the half-warps, then a
// reduce-scatter (31 shuffles for 16 sums)
__device__ __forceinline__ double warp_reduce_scatter16(double (&acc)[16], int lane) {
#pragma unroll
  for (int k = 0; k < 16; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 16);
#pragma unroll
  for (int s = 8; s >= 1; s >>= 1) {
    const bool up = (lane & s) != 0;
#pragma unroll
    for (int k = 0; k < s; ++k) {
      const double send = up ? acc[k] : acc[k + s];
      const double keep = up ? acc[k + s] : acc[k];
      acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
  }
  return acc[0];
}

__global__ void __launch_bounds__(TT)
tridiag_blocked_cluster(const EigDev* __restrict__ probs, double* G, double* Tg, double* VWg) {
  extern __shared__ double sm[];
  __shared__ double red[33];
  __shared__ double s_K;
  __shared__ double vw_part[NWARP * 2 * PNB_MAX];  // per-warp V^T v, W^T v sums

  cgx::cluster_group cluster = cgx::this_cluster();
  const int CL = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const EigDev P = probs[blockIdx.x / CL];
  const int n = P.n;
  const int tid = threadIdx.x;
  if (n <= 0) return;  // the same problem for the whole cluster
  const int nb = P.nb;
  double* Gp = G + P.g_off;
  double* dg = Tg + 3 * P.w_off;
  double* eg = dg + n;
  double* tg = eg + n;
  double* VW = VWg + P.s_off;  // n x 2nb, row-major: [i][t] = V(i, t), [i][nb + t] = W(i, t)
  const int warp = tid >> 5, lane = tid & 31;
  const int nloc = (n + CL - 1) / CL;
  int lown = 0;  // own indices c = rank + CL l, l < lown
  while (lown < nloc && rank + CL * lown < n) ++lown;
  double* Vl = sm;                            // [nb][nloc]
  double* Wl = Vl + (int64_t)nb * nloc;       // [nb][nloc]
  double* xc = Wl + (int64_t)nb * nloc;       // [2][nloc]: own rows of a column, by parity of jj
  // Vectors over all rows are kept owner-major: row i = r + CL l at [r nloc + l],
  // so what one CTA pushes to another is contiguous on both sides
  const int lg = __ffs(CL) - 1;  // CL is a power of two
  auto om = [&](int i) { return ((i & (CL - 1)) * nloc) + (i >> lg); };
  double* xo = xc + 2 * nloc;                 // [CL][nloc]: column j as pushed, then v
  double* yl = xo + (int64_t)CL * nloc;       // [CL][nloc]: this CTA's row sums of A22 v
  double* yb = yl + (int64_t)CL * nloc;       // [CL][nloc]: row sums of A22 v on the own rows, by sender
  double* dw = yb + (int64_t)CL * nloc;       // [NWARP][nloc]: column dots by warp
  double* r2 = dw + (int64_t)NWARP * nloc;    // [CL_MAX][2nb]: V^T v, W^T v partials by sender
  double* r3 = r2 + CL_MAX * 2 * nb;          // [CL_MAX]: v^T A22 v partials by sender
  double* yp = r3 + CL_MAX;                   // [CL_MAX][nb]: row sums on the panel's rows by sender
  double* dp = yp + CL_MAX * nb;              // [nb]: column dots of the panel's rows
  double* Vp = dp + nb;                       // [nb][nb]: Vp[t nb + s] = v_t[k0 + s]
  double* Wq = Vp + nb * nb;                  // [nb][nb]: Wq[t nb + s] = w_t[k0 + s]
  double* cvt = Wq + nb * nb;                 // [nb]: V^T v
  double* cwt = cvt + nb;                     // [nb]: W^T v
  for (int k0 = 0; k0 + 2 < n; k0 += nb) {
    const int nbe = min(nb, n - 2 - k0);  // reflector columns k0 .. k0 + nbe - 1
    for (int jj = 0; jj < nbe; ++jj) {
      const int j = k0 + jj;
      double* xcur = xc + (jj & 1) * nloc;
      // ---- 1: column j on the own rows >= j, pushed to every CTA ----
      const int l1 = first_owned(j, rank, CL);
      {
        // four threads per row, each summing a quarter of the panel's terms
        // (the loop bound is the same for the whole warp: the shuffles need it)
        const int sub = tid & 3;
        for (int base = l1 + (warp << 3); base < lown; base += blockDim.x >> 2) {
          const int l = base + (lane >> 2);
          const bool act = l < lown;
          double corr = 0.0;
          if (act)
#pragma unroll 1
            for (int t = sub; t < jj; t += 4)
              corr += Vl[t * nloc + l] * Wq[t * nb + jj] + Wl[t * nloc + l] * Vp[t * nb + jj];
          corr += __shfl_xor_sync(0xffffffffu, corr, 1);
          corr += __shfl_xor_sync(0xffffffffu, corr, 2);
          if (act && sub == 0) xcur[l] = (jj == 0 ? Gp[(rank + CL * l) + (int64_t)n * j] : xcur[l]) - corr;
        }
      }
      __syncthreads();
      for (int e = tid; e < (lown - l1) * CL; e += blockDim.x) {
        const int q = e / (lown - l1), l = l1 + e % (lown - l1);
        *cluster.map_shared_rank(xo + rank * nloc + l, q) = xcur[l];
      }
      cluster.sync();  // A
      // ---- 2: the reflector (same in every CTA), v kept, V^T v and W^T v partials ----
      const double alpha = xo[om(j + 1)];  // read before the reduction's barriers, overwritten below
      double part = 0.0;
      for (int i = j + 2 + tid; i < n; i += blockDim.x) part += xo[om(i)] * xo[om(i)];
      const double sigma = block_reduce(part, red, false);
      double tau = 0.0, beta = alpha, scale = 0.0;
      if (sigma != 0.0) {
        const double mu = sqrt(alpha * alpha + sigma);
        beta = alpha <= 0.0 ? mu : -mu;
        tau = (beta - alpha) / beta;
        scale = 1.0 / (alpha - beta);
      }
      if (rank == j % CL && tid == 0) {
        dg[j] = xo[om(j)];
        tg[j] = tau;
        eg[j] = beta;
      }
      for (int i = j + 1 + tid; i < n; i += blockDim.x) xo[om(i)] = i == j + 1 ? 1.0 : xo[om(i)] * scale;
      __syncthreads();
      for (int l = tid; l < lown; l += blockDim.x) {
        const int i = rank + CL * l;
        const double vi = i >= j + 1 ? xo[rank * nloc + l] : 0.0;
        Vl[jj * nloc + l] = vi;
        Wl[jj * nloc + l] = 0.0;
        if (i >= j + 2) Gp[i + (int64_t)n * j] = vi;  // reflector kept below the subdiagonal for phase 2
      }
      for (int s = tid; s < nb; s += blockDim.x) {
        const int row = k0 + s;
        Vp[jj * nb + s] = row >= j + 1 && row < n ? xo[om(row)] : 0.0;
      }
      __syncthreads();
      const int lf = first_owned(j + 1, rank, CL);
      // V^T v and W^T v partials over the own rows >= j + 1: lane t of each
      // warp sums column t over every NWARP-th row, the warps' sums are added
      // in warp order and pushed to every CTA
      if (jj > 0) {
        double sv = 0.0, sw = 0.0;
        if (lane < jj)
          for (int l = lf + warp; l < lown; l += NWARP) {
            const double v = Vl[jj * nloc + l];
            sv += Vl[lane * nloc + l] * v;
            sw += Wl[lane * nloc + l] * v;
          }
        vw_part[warp * 2 * PNB_MAX + lane] = sv;
        vw_part[warp * 2 * PNB_MAX + PNB_MAX + lane] = sw;
        __syncthreads();
        if (tid < 2 * PNB_MAX) {
          const int t = tid & (PNB_MAX - 1);
          if (t < jj) {
            double a = 0.0;
            for (int w = 0; w < NWARP; ++w) a += vw_part[w * 2 * PNB_MAX + tid];
            const int slot = rank * 2 * nb + (tid < PNB_MAX ? t : nb + t);
            for (int q = 0; q < CL; ++q) *cluster.map_shared_rank(r2 + slot, q) = a;
          }
        }
      }
      // ---- 3: p = A22 v from the lower triangle of the own columns ----
      if (jj + 1 < nbe)  // the next column's own rows: unchanged until its step 1
        for (int l = lf + tid; l < lown; l += blockDim.x)
          xc[((jj + 1) & 1) * nloc + l] = Gp[(rank + CL * l) + (int64_t)n * (j + 1)];
      double kp = 0.0;  // this thread's share of v^T A22 v
      if (tau != 0.0) {
        for (int l = lf + lane; l < lown; l += 32) dw[warp * nloc + l] = 0.0;
        __syncwarp();
        // blocks of 64 rows from row j + 1, two rows per lane (i0 = rb + lane,
        // i1 = i0 + 32); the longest (last) blocks are dealt first and back and
        // forth, so the warps' shares come out even
        const int nrb = (n - j - 1 + 63) / 64;
        const int64_t cstep = (int64_t)n * CL;  // from one own column to the next
        for (int round = 0; round * NWARP < nrb; ++round) {
          const int o = round * NWARP + ((round & 1) ? NWARP - 1 - warp : warp);
          if (o >= nrb) continue;
          const int rb = j + 1 + 64 * (nrb - 1 - o);
          const int i0 = rb + lane, i1 = i0 + 32;
          const double v0 = i0 < n ? xo[om(i0)] : 0.0, v1 = i1 < n ? xo[om(i1)] : 0.0;
          // rows past the end read row n - 1 (weighted by v = 0, sums discarded)
          const double* g0 = Gp + min(i0, n - 1) + (int64_t)n * rank;
          const double* g1 = Gp + min(i1, n - 1) + (int64_t)n * rank;
          const int le = first_owned(min(n, rb + 64), rank, CL);  // own columns c < the block's end
          const int lfull = min(le, first_owned(rb, rank, CL));   // own columns c < rb: no masking
          double y0 = 0.0, y1 = 0.0;
          int lt = lf;
          for (; lt + 16 <= lfull; lt += 16) {
            double acc[16];
#pragma unroll
            for (int h = 0; h < 16; h += 8) {  // eight columns' loads in flight at a time
              double a0[8], a1[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                a0[k] = g0[(lt + h + k) * cstep];
                a1[k] = g1[(lt + h + k) * cstep];
              }
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const double vc = xo[rank * nloc + lt + h + k];
                y0 = fma(a0[k], vc, y0);
                y1 = fma(a1[k], vc, y1);
                acc[h + k] = fma(a1[k], v1, a0[k] * v0);
              }
            }
            const double d = warp_reduce_scatter16(acc, lane);
            if (lane < 16) dw[warp * nloc + lt + lane] += d;
          }
          for (; lt < le; lt += 16) {  // the rest, masked: the block's diagonal part and a short tail
            double acc[16];
#pragma unroll
            for (int h = 0; h < 16; h += 8) {
              double a0[8], a1[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const int c = rank + CL * (lt + h + k);
                const bool cv = lt + h + k < le;
                a0[k] = cv && i0 >= c ? g0[(lt + h + k) * cstep] : 0.0;
                a1[k] = cv && i1 >= c ? g1[(lt + h + k) * cstep] : 0.0;
              }
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const int c = rank + CL * (lt + h + k);
                const double vc = lt + h + k < le ? xo[rank * nloc + lt + h + k] : 0.0;
                y0 = fma(i0 > c ? a0[k] : 0.0, vc, y0);
                y1 = fma(i1 > c ? a1[k] : 0.0, vc, y1);
                acc[h + k] = fma(a1[k], v1, a0[k] * v0);
              }
            }
            const double d = warp_reduce_scatter16(acc, lane);
            if (lane < 16 && lt + lane < le) dw[warp * nloc + lt + lane] += d;
          }
          if (i0 < n) {
            yl[om(i0)] = y0;
            kp += v0 * y0;
          }
          if (i1 < n) {
            yl[om(i1)] = y1;
            kp += v1 * y1;
          }
        }
      }
      __syncthreads();
      if (tau != 0.0) {
        // the row sums to their owners (rows below j + 1 and beyond n ride
        // along unread), those of the panel's rows to every CTA
        const int lmin = (j + 1) >> lg, cnt = nloc - lmin;
        for (int e = tid; e < CL * cnt; e += blockDim.x) {
          const int d = e / cnt, l = lmin + e % cnt;
          *cluster.map_shared_rank(yb + rank * nloc + l, d) = yl[d * nloc + l];
        }
        for (int e = tid; e < CL * nb; e += blockDim.x) {
          const int q = e / nb, s = e % nb, row = k0 + s;
          if (row >= j + 1 && row < n) *cluster.map_shared_rank(yp + rank * nb + s, q) = yl[om(row)];
        }
      }
      if (tau != 0.0)
        for (int l = lf + tid; l < lown; l += blockDim.x) {
          double d = 0.0;
          for (int w = 0; w < NWARP; ++w) d += dw[w * nloc + l];
          dw[l] = d;  // the column's dot, kept in warp 0's row
          const int c = rank + CL * l;
          kp += xo[rank * nloc + l] * d;
          if (c < k0 + nb)
            for (int q = 0; q < CL; ++q) *cluster.map_shared_rank(dp + (c - k0), q) = d;
        }
      const double vav_part = block_reduce(kp, red, false);
      if (tid < CL) *cluster.map_shared_rank(r3 + rank, tid) = vav_part;
      cluster.sync();  // B
      // ---- 4: w on the own rows and on the panel's rows ----
      if (warp == 0) {  // V^T v, W^T v and the scalar K = (tau/2) w'.v, one lane per panel column
        double a = 0.0, b = 0.0;
        if (lane < jj)
          for (int q = 0; q < CL; ++q) {
            a += r2[q * 2 * nb + lane];
            b += r2[q * 2 * nb + nb + lane];
          }
        if (lane < jj) {
          cvt[lane] = a;
          cwt[lane] = b;
        }
        const double cc = warp_sum(a * b);
        if (lane == 0) {
          double vav = 0.0;
          for (int q = 0; q < CL; ++q) vav += r3[q];
          s_K = 0.5 * tau * tau * (vav - 2.0 * cc);
        }
      }
      __syncthreads();
      if (tau != 0.0) {
        const double K = s_K;
        // own rows: four threads per row, each summing a quarter of the terms
        // (the loop bound is the same for the whole warp: the shuffles need it)
        const int sub = tid & 3;
        for (int base = lf + (warp << 3); base < lown; base += blockDim.x >> 2) {
          const int l = base + (lane >> 2);
          const bool act = l < lown;
          double p = 0.0, corr = 0.0;
          if (act) {
#pragma unroll 1
            for (int q = sub; q < CL; q += 4) p += yb[q * nloc + l];
#pragma unroll 1
            for (int t = sub; t < jj; t += 4) corr += Vl[t * nloc + l] * cwt[t] + Wl[t * nloc + l] * cvt[t];
          }
          p += __shfl_xor_sync(0xffffffffu, p, 1);
          p += __shfl_xor_sync(0xffffffffu, p, 2);
          corr += __shfl_xor_sync(0xffffffffu, corr, 1);
          corr += __shfl_xor_sync(0xffffffffu, corr, 2);
          if (act && sub == 0) Wl[jj * nloc + l] = tau * (dw[l] + p - corr) - K * Vl[jj * nloc + l];
        }
        // the panel's rows: sixteen threads per row
        const int s = tid >> 4, sub16 = tid & 15;
        if (s < nb) {
          const int row = k0 + s;
          const bool live = row >= j + 1 && row < n;
          double p = 0.0, corr = 0.0;
          if (live) {
            for (int q = sub16; q < CL; q += 16) p += yp[q * nb + s];
            for (int t = sub16; t < jj; t += 16) corr += Vp[t * nb + s] * cwt[t] + Wq[t * nb + s] * cvt[t];
          }
#pragma unroll
          for (int o = 1; o < 16; o <<= 1) {
            p += __shfl_xor_sync(0xffffffffu, p, o);
            corr += __shfl_xor_sync(0xffffffffu, corr, o);
          }
          if (sub16 == 0) Wq[jj * nb + s] = live ? tau * (dp[s] + p - corr) - K * Vp[jj * nb + s] : 0.0;
        }
      } else {
        for (int s = tid; s < nb; s += blockDim.x) Wq[jj * nb + s] = 0.0;
      }
      __syncthreads();
    }
    // ---- trailing update A[k1:, k1:] -= V W^T + W V^T (lower triangle) through the global scratch ----
    const int k1 = k0 + nbe;
    for (int e = tid; e < lown * 2 * nbe; e += blockDim.x) {
      const int l = e / (2 * nbe), t2 = e - l * 2 * nbe;
      const int i = rank + CL * l;
      if (i < k1) continue;
      const int t = t2 < nbe ? t2 : t2 - nbe;
      VW[(int64_t)i * 2 * nb + (t2 < nbe ? t : nb + t)] = (t2 < nbe ? Vl : Wl)[t * nloc + l];
    }
    __threadfence();
    cluster.sync();
    // DMMA (m8n8k4 f64) tiles: a warp takes 32 rows x 16 own columns and runs
    // P = V W^T + W V^T over the panel's k, the rows' [V W] fragments read
    // straight from the scratch (no shared staging, no barrier per tile); the
    // lower triangle of its block then receives A -= P
    const int lf = first_owned(k1, rank, CL);
    const int nbe4 = (nbe + 3) & ~3;
    const int gr = lane >> 2, gk = lane & 3;
    const int nrt = (n - k1 + 31) >> 5;                 // 32-row tiles
    const int ncb = (first_owned(n, rank, CL) - lf + 15) >> 4;  // 16-column blocks
    for (int task = warp; task < nrt * ncb; task += NWARP) {
      const int i0 = k1 + 32 * (task / ncb), lb = lf + 16 * (task % ncb);
      if (rank + CL * lb > i0 + 31) continue;  // the block lies above the diagonal
      const int le = min(first_owned(min(n, i0 + 32), rank, CL), lb + 16);
      double acc[4][2][2];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        // part 0: V (rows) x W (columns); part 1: W x V
        const int xo0 = part ? nb : 0;
        const double* Y = part ? Vl : Wl;
#pragma unroll 1
        for (int t = 0; t < nbe4; t += 4) {
          const int k = t + gk;
          const bool kv = k < nbe;
          double af[4], bf[2];
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const int i = i0 + 8 * a + gr;
            af[a] = kv && i < n ? VW[(int64_t)i * 2 * nb + xo0 + k] : 0.0;
          }
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const int l = lb + 8 * b + gr;
            bf[b] = kv && l < le ? Y[k * nloc + l] : 0.0;
          }
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) dmma_tr(acc[a][b], af[a], bf[b]);
        }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int i = i0 + 8 * a + gr;
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int l = lb + 8 * b + 2 * gk + e;
            const int c = rank + CL * l;
            if (i < n && l < le && i >= c) Gp[(int64_t)n * c + i] -= acc[a][b][e];
          }
      }
    }
    __threadfence();
    cluster.sync();
  }
  // T: the last two diagonal entries and the last off-diagonal A[n-1, n-2]
  if (tid == 0) {
    if (rank == (n - 2) % CL) {
      dg[n - 2] = Gp[(n - 2) + (int64_t)n * (n - 2)];
      eg[n - 2] = Gp[(n - 1) + (int64_t)n * (n - 2)];
    }
    if (rank == (n - 1) % CL) dg[n - 1] = Gp[(n - 1) + (int64_t)n * (n - 1)];
    if (rank == 0) {
      eg[n - 1] = 0.0;
      tg[n - 1] = 0.0;
      tg[n - 2] = 0.0;
    }
  }
  __threadfence();
  cluster.sync();  // also the last access of another CTA's shared memory
}

// Bisection for every sector after its tridiagonalisation, spread over the
// GPU: a CTA of BS_THREADS threads takes BS_PER eigenvalues of one problem, with
// the problem's d and e^2 in shared memory, scaled by a power of two to a norm in
// [1/2, 1).  Sixteen lanes serve one eigenvalue: in a round they count at the 15
// points that four successive halvings of the current interval can probe (the
// nodes of a four-level bisection tree, each computed by the same chain of
// midpoints that plain bisection would compute), then every lane of the group
// walks the tree with the shared counts.  The intervals and the stopping rule
// are those of plain bisection; a round advances four halvings instead of one,
// so an eigenvalue takes about 13 rounds of Sturm chains instead of 50.
// Bound by the FP64 pipe where there are many eigenvalues (three operations a
// step and lane), by the chain of FMAs where there are few.  All sectors of a
// block SVD at bond dimension 3072: 1977 (those above 160 only) -> 626 us.
constexpr int BS_THREADS = 128;
constexpr int BS_LANES = 16;  // lanes per eigenvalue: 15 probes, one idle
constexpr int BS_LEVELS = 4;  // halvings per round
constexpr int BS_PER = BS_THREADS / BS_LANES;

__global__ void __launch_bounds__(BS_THREADS)
bisect_sectors(const EigDev* __restrict__ probs, const VecTaskB* __restrict__ tasks, const double* Tg, double* W) {
  extern __shared__ double bs_sm[];
  __shared__ double red[33];
  const VecTaskB tk = tasks[blockIdx.x];
  const EigDev P = probs[tk.prob];
  const int n = P.n;
  const double* dg = Tg + 3 * P.w_off;
  const double* eg = dg + n;
  double* Wp = W + P.w_off;
  const int tid = threadIdx.x, lane = tid & 31;
  double2* de = reinterpret_cast<double2*>(bs_sm);
  const int npad = (n + 7) & ~7;
  // Gershgorin bounds
  double lo_loc = DBL_MAX, hi_loc = -DBL_MAX;
  for (int i = tid; i < n; i += blockDim.x) {
    const double r = (i > 0 ? fabs(eg[i - 1]) : 0.0) + (i < n - 1 ? fabs(eg[i]) : 0.0);
    lo_loc = fmin(lo_loc, dg[i] - r);
    hi_loc = fmax(hi_loc, dg[i] + r);
  }
  double gu = block_reduce(hi_loc, red, true);
  double gl = -block_reduce(-lo_loc, red, true);
  double bnorm = fmax(fabs(gl), fabs(gu));
  if (!(bnorm > 0.0) || !isfinite(bnorm)) {  // T == 0: every eigenvalue is exactly zero (not finite: passed on)
    for (int j = tk.j0 + tid; j < min(n, tk.j0 + BS_PER); j += blockDim.x) Wp[n - 1 - j] = bnorm;
    return;
  }
  int ex;
  frexp(bnorm, &ex);
  const double sc = ldexp(1.0, -max(ex, -1000)), isc = ldexp(1.0, max(ex, -1000));
  gu *= sc;
  gl *= sc;
  bnorm *= sc;
  for (int i = tid; i < npad; i += blockDim.x) {
    const double ei = i > 0 && i < n ? eg[i - 1] * sc : 0.0;
    de[i] = i < n ? make_double2(dg[i] * sc, i > 0 ? fmax(ei * ei, STURM_E2) : 0.0) : make_double2(4.0, 0.0);
  }
  __syncthreads();
  const double atol = 4.0 * DBL_EPSILON * bnorm;
  auto open_interval = [&](double lo, double hi) {
    return hi - lo > fmax(atol, 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)));
  };
  const int sub = lane & (BS_LANES - 1);          // this lane's tree node: in-order position sub + 1
  const int base = lane & ~(BS_LANES - 1);        // first lane of the group
  const int j = tk.j0 + tid / BS_LANES;
  const bool active = j < n;
  constexpr int ROOT = 1 << (BS_LEVELS - 1);      // in-order position of the root (8)
  double lo = gl - atol, hi = gu + atol;
  int it = 0;
  bool work = active && open_interval(lo, hi);
  while (__any_sync(0xffffffffu, work)) {
    int c = 0;
    if (work && sub < 2 * ROOT - 1) {
      // descend from the round's interval to node sub + 1 by midpoints
      const int p = sub + 1;
      double a = lo, b = hi;
      int pos = ROOT, half = ROOT >> 1;
      while (pos != p) {
        const double m = 0.5 * (a + b);
        if (p < pos) { b = m; pos -= half; } else { a = m; pos += half; }
        half >>= 1;
      }
      c = sturm_count(de, npad, 0.5 * (a + b));
    }
    // every lane of the group walks the same path with the group's counts
    int pos = ROOT, half = ROOT >> 1;
    bool go = work;
#pragma unroll
    for (int lev = 0; lev < BS_LEVELS; ++lev) {
      const int cp = __shfl_sync(0xffffffffu, c, base + pos - 1);
      go = go && it < 128 && open_interval(lo, hi);
      if (go) {
        const double mid = 0.5 * (lo + hi);
        if (cp > j) { hi = mid; pos -= half; } else { lo = mid; pos += half; }
        half >>= 1;
        ++it;
      }
    }
    if (work) work = it < 128 && open_interval(lo, hi);
  }
  if (active && sub == 0) Wp[n - 1 - j] = 0.5 * (lo + hi) * isc;
}

__global__ void __launch_bounds__(TT)
tridiag_eigvecs_cluster(const EigDev* __restrict__ probs, const double* G, const double* Tg, const double* W,
                        double* Zg, double* work, int cap, const int* __restrict__ only_flagged) {
  extern __shared__ double zsm[];
  __shared__ double red[33];
  __shared__ double coef[MAX_N / 2];
  __shared__ int cstart[MAX_N / 2];
  cgx::cluster_group cluster = cgx::this_cluster();
  const int CL = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  // as the fallback of the blocked path: only the problems it flagged (the
  // whole cluster returns alike, before any barrier)
  if (only_flagged && only_flagged[blockIdx.x / CL] == 0) return;
  const EigDev P = probs[blockIdx.x / CL];
  const int n = P.n, nvec = P.nvec;
  const int tid = threadIdx.x;
  if (n <= 0 || nvec <= 0) return;  // the same problem for the whole cluster
  double* Zout = Zg + P.g_off;
  const int q = (nvec + CL - 1) / CL;
  const int j0 = rank * q, j1 = min(nvec, j0 + q), nown = max(0, j1 - j0);
  const bool in_smem = (int64_t)q * n + 6 * (int64_t)n <= cap;
  double* Z = in_smem ? zsm : Zout + (int64_t)n * j0;  // own vector t at Z + n t
  double* ybuf = in_smem ? zsm + (int64_t)q * n : zsm;  // the current Gram-Schmidt iterate
  double* ubuf = ybuf + n;                              // [2][n] published partial projections
  double* scr = ubuf + 2 * n;                           // 3n LU scratch
  const double* d = Tg + 3 * P.w_off;
  const double* e = d + n;
  const double* tau = e + n;
  const double* lam = W + P.w_off;  // descending
  const double* Gp = G + P.g_off;
  const int warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  double loc = 0.0;
  for (int i = tid; i < n; i += blockDim.x)
    loc = fmax(loc, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
  const double tnorm = block_reduce(loc, red, true);
  const double tiny = tnorm > 1e-250 ? fmax(DBL_EPSILON * tnorm, DBL_MIN) : 1.0;
  const double ortol = 1e-3 * tnorm;
  // (a) inverse iteration on the own vectors, one thread each (same start vectors as the one-CTA kernel)
  for (int t = tid; t < nown; t += blockDim.x) {
    const int j = j0 + t;
    double* y = Z + (int64_t)n * t;
    for (int i = 0; i < n; ++i) y[i] = hash_unit(((uint64_t)P.g_off << 20) ^ ((uint64_t)j << 32) ^ (uint64_t)i);
    for (int it = 0; it < INV_ITERS; ++it) {
      tri_solve(d, e, n, lam[j], tiny, y, work + 3 * P.g_off + (int64_t)3 * n * j, 1);
      double s = 0.0;
      for (int i = 0; i < n; ++i) s += y[i] * y[i];
      const double inv = 1.0 / sqrt(s);
      for (int i = 0; i < n; ++i) y[i] *= inv;
    }
  }
  if (tid == 0) {
    int c = 0;
    for (int j = 0; j < nvec && j < MAX_N / 2; ++j) {
      if (j == 0 || lam[j - 1] - lam[j] > ortol) c = j;
      cstart[j] = c;
    }
  }
  __syncthreads();
  cluster.sync();  // every start vector is in place
  // (b) Gram-Schmidt, vector by vector.  Which CTAs hold members of the
  // cluster [c0, j) follows from c0, j and q alone, so no flags are exchanged;
  // every CTA holds the same iterate y and forms its norm in the same order.
  int g = 0;
  for (int j = 1; j < nvec && j < MAX_N / 2; ++j) {
    const int c0 = cstart[j];
    if (c0 == j) continue;
    const int owner = j / q;
    const double* yj = in_smem ? cluster.map_shared_rank(zsm + (int64_t)n * (j - owner * q), owner)
                               : Zout + (int64_t)n * j;
    __syncthreads();  // every read of the previous iterate is done
    for (int i = tid; i < n; i += blockDim.x) ybuf[i] = yj[i];
    __syncthreads();
    const int ka = max(c0, j0), kb = min(j, j1);  // own members of the cluster before j
    const int o_lo = c0 / q, o_hi = (j - 1) / q;  // CTAs that own members
    for (int pass = 0; pass < 6; ++pass) {
      double n0 = 0.0;  // |y|^2 before the projections, every warp alike
      for (int i = lane; i < n; i += 32) n0 += ybuf[i] * ybuf[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) n0 += __shfl_xor_sync(0xffffffffu, n0, o);
      for (int r = 0; r < 2; ++r) {
        const int par = g & 1;
        double* u = ubuf + par * n;
        for (int k = ka + warp; k < kb; k += nw) {
          const double* __restrict__ zk = Z + (int64_t)n * (k - j0);
          double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;  // independent chains
          int i = lane;
          for (; i + 96 < n; i += 128) {
            s0 += zk[i] * ybuf[i];
            s1 += zk[i + 32] * ybuf[i + 32];
            s2 += zk[i + 64] * ybuf[i + 64];
            s3 += zk[i + 96] * ybuf[i + 96];
          }
          for (; i < n; i += 32) s0 += zk[i] * ybuf[i];
          double s = (s0 + s1) + (s2 + s3);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
          if (lane == 0) coef[k - ka] = s;
        }
        __syncthreads();
        if (kb > ka)
          for (int i = tid; i < n; i += blockDim.x) {
            const double* __restrict__ zi = Z + (int64_t)n * (ka - j0) + i;
            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
            int k = 0;
            const int nk = kb - ka;
            for (; k + 3 < nk; k += 4) {
              s0 += coef[k] * zi[(int64_t)n * k];
              s1 += coef[k + 1] * zi[(int64_t)n * (k + 1)];
              s2 += coef[k + 2] * zi[(int64_t)n * (k + 2)];
              s3 += coef[k + 3] * zi[(int64_t)n * (k + 3)];
            }
            for (; k < nk; ++k) s0 += coef[k] * zi[(int64_t)n * k];
            u[i] = (s0 + s1) + (s2 + s3);
          }
        cluster.sync();
        for (int i = tid; i < n; i += blockDim.x) {
          double rr[CL_MAX];  // every remote load in flight at once, then the sum in CTA order
#pragma unroll
          for (int o = 0; o < CL_MAX; ++o)
            rr[o] = (o >= o_lo && o <= o_hi && o < CL) ? *cluster.map_shared_rank(u + i, o) : 0.0;
          double s = ybuf[i];
#pragma unroll
          for (int o = 0; o < CL_MAX; ++o) s -= rr[o];
          ybuf[i] = s;
        }
        __syncthreads();
        ++g;
        if (r == 0) {
          // "twice is enough" (Kahan, Parlett): a second projection only when
          // the first removed more than half of |y|^2; every CTA and warp holds
          // the same y and takes the same decision
          double n1 = 0.0;
          for (int i = lane; i < n; i += 32) n1 += ybuf[i] * ybuf[i];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) n1 += __shfl_xor_sync(0xffffffffu, n1, o);
          if (n1 > 0.5 * n0) break;
        }
      }
      double nl = 0.0;  // every warp: the whole norm, same order
      for (int i = lane; i < n; i += 32) nl += ybuf[i] * ybuf[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) nl += __shfl_xor_sync(0xffffffffu, nl, o);
      const double nrm = sqrt(nl);
      if (nrm > 0.5 || pass == 5) {
        const double inv = nrm > 0.0 ? 1.0 / nrm : 0.0;
        if (rank == owner)
          for (int i = tid; i < n; i += blockDim.x) Z[(int64_t)n * (j - j0) + i] = ybuf[i] * inv;
        break;
      }
      // collapsed onto earlier vectors: one more inverse iteration from the
      // orthogonal remainder (every CTA alike), then orthogonalise again
      __syncthreads();
      if (tid == 0) {
        const double inv = nrm > 0.0 ? 1.0 / nrm : 1.0;
        for (int i = 0; i < n; ++i) ybuf[i] = nrm > 0.0 ? ybuf[i] * inv : hash_unit((uint64_t)(j * 7919 + i + pass));
        tri_solve(d, e, n, lam[j], tiny, ybuf, scr, 1);
      }
      __syncthreads();
    }
  }
  cluster.sync();  // no CTA reads another's shared memory after this point
  // (c) back-transformation z = H_0 H_1 ... H_{n-3} y, last reflector first
  double* stg = ubuf;  // CL_STAGE staged reflectors (5n doubles available)
  for (int kb = n - 3; kb >= 0; kb -= CL_STAGE) {
    __syncthreads();
    for (int s = 0; s < CL_STAGE && kb - s >= 0; ++s) {
      const int k = kb - s, m = n - k - 1;
      for (int i = tid; i < m; i += blockDim.x) stg[(int64_t)s * n + i] = (i == 0) ? 1.0 : Gp[(k + 1 + i) + (int64_t)n * k];
    }
    __syncthreads();
    for (int t = warp; t < nown; t += nw) {
      double* y = Z + (int64_t)n * t;
      for (int s = 0; s < CL_STAGE && kb - s >= 0; ++s) {
        const int k = kb - s, m = n - k - 1;
        const double tk = tau[k];
        if (tk == 0.0) continue;
        const double* __restrict__ v = stg + (int64_t)s * n;
        const double* __restrict__ yk = y + k + 1;
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;  // independent chains
        int i = lane;
        for (; i + 96 < m; i += 128) {
          a0 += v[i] * yk[i];
          a1 += v[i + 32] * yk[i + 32];
          a2 += v[i + 64] * yk[i + 64];
          a3 += v[i + 96] * yk[i + 96];
        }
        for (; i < m; i += 32) a0 += v[i] * yk[i];
        double acc = (a0 + a1) + (a2 + a3);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        const double c = tk * acc;
        for (int i = lane; i < m; i += 32) y[k + 1 + i] -= v[i] * c;
        __syncwarp();
      }
    }
  }
  __syncthreads();
  // (d) deterministic gauge: the largest-magnitude entry (first on ties) is positive
  for (int t = warp; t < nown; t += nw) {
    double* y = Z + (int64_t)n * t;
    double best = -1.0;
    int bi = n;
    for (int i = lane; i < n; i += 32) {
      const double a = fabs(y[i]);
      if (a > best) { best = a; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    const bool flip = bi < n && y[bi] < 0.0;
    __syncwarp();
    if (flip)
      for (int i = lane; i < n; i += 32) y[i] = -y[i];
  }
  if (in_smem) {
    __syncthreads();
    for (int64_t i = tid; i < (int64_t)n * nown; i += blockDim.x) Zout[(int64_t)n * j0 + i] = Z[i];
  }
}

// ---------------------------------------------------------------------------
// Eigenvectors of the cluster-sized sectors, across the whole GPU.
//
// (1) inverse iteration, one thread per wanted vector (same start vectors and
//     solves as the kernels above);
// (2) CholeskyQR2 (Fukaya et al., "CholeskyQR2: a simple and communication-
//     avoiding algorithm", 2014): G = Z^T Z, G = L L^T, Z <- Z L^-T, twice.
//     In exact arithmetic this is Gram-Schmidt in column (descending
//     eigenvalue) order, i.e. what the kernels above do inside clusters of
//     close eigenvalues; against the other vectors it only removes components
//     of the size of their orthogonality error.  A pivot L_jj below 1e-4 in
//     the first pass means vector j had collapsed onto earlier ones (its
//     orthonormalised form would carry a residual of eps ||T|| / L_jj): the
//     problem is flagged and the cluster kernel above, which re-iterates such
//     vectors, redoes it from the start;
// (3) back-transformation z = Q y with the reflectors grouped 32 at a time in
//     the compact WY form Q_p = I - V T V^T (LAPACK dlarft, forward and
//     columnwise), then the deterministic gauge.
// Every launch is batched over the problems; (1)-(3) use as many CTAs as
// there are vectors, rows or tiles.
constexpr int IV_THREADS = 32;    // vectors per CTA of the inverse iteration
constexpr int GT = 64;            // Gram tile
constexpr int CH_PB = 32;         // Cholesky panel
constexpr int CH_THREADS = 256;   // threads per CTA of the Cholesky: 255 registers hold a tile and all its fragments
constexpr int CH_LD = CH_PB + 2;  // leading dimension of its triangle in shared memory
constexpr int TS_ROWS = 32;       // rows per CTA of the triangular solve
constexpr int TS_THREADS = 128;   // its threads: two CTAs of 255 registers per SM
constexpr int BT_NB = 32;         // reflectors per compact-WY panel
constexpr int BT_VB = 16;         // vectors per CTA of the back-transformation
constexpr double COLLAPSE_PIVOT2 = 1e-8;  // L_jj^2 below this: collapsed vector
__device__ unsigned long long g_eig_redo;  // problems whose vectors the cluster kernel redid (device-wide)

struct VecTask {
  int32_t prob, j0;  // problem (index into the problem array) and first item
};
struct TileTask {
  int32_t prob, a, b;  // problem and tile / panel coordinates
};

__device__ double tnorm1(const double* d, const double* e, int n, double* red) {
  double loc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    loc = fmax(loc, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
  return block_reduce(loc, red, true);
}

// (1) inverse iteration: thread t of task (p, j0) computes vector j0 + t
__global__ void __launch_bounds__(IV_THREADS)
inv_iter_batched(const EigDev* __restrict__ probs, const VecTask* __restrict__ tasks, const double* Tg,
                 const double* W, double* Zg, double* work) {
  extern __shared__ double de[];  // T: d and e
  __shared__ double red[33];
  const VecTask tk = tasks[blockIdx.x];
  const EigDev P = probs[tk.prob];
  const int n = P.n;
  double *d = de, *e = de + n;
  for (int i = threadIdx.x; i < 2 * n; i += IV_THREADS) de[i] = i < 2 * n - 1 ? Tg[3 * P.w_off + i] : 0.0;
  __syncthreads();
  const double* lam = W + P.w_off;
  const double tnorm = tnorm1(d, e, n, red);
  const double tiny = tnorm > 1e-250 ? fmax(DBL_EPSILON * tnorm, DBL_MIN) : 1.0;
  const int t = threadIdx.x, j = tk.j0 + t;
  const int cnt = min(IV_THREADS, P.nvec - tk.j0);  // vectors of this CTA
  const bool active = t < cnt;  // no early return: the barrier below needs every thread
  // the CTA's iterates and factors interleaved (element i of its vector t at
  // [i cnt + t]), so that the threads' accesses coalesce: the iterates, u0 and u1
  // in the problem's work area (3 n cnt doubles from work + 3 g_off + 3 n j0), the
  // multipliers in the CTA's own columns of Z (n cnt doubles), which receive the
  // vectors at the end
  double* wb = work + 3 * P.g_off + (int64_t)3 * n * tk.j0;
  double* zb = Zg + P.g_off + (int64_t)n * tk.j0;
  double* y = wb + t;
  const int64_t nc = (int64_t)n * cnt;
  // each iterate's normalisation is applied as the next solve (or the final
  // copy) reads it; its norm is summed in the solve's back substitution
  double inv = 1.0;
  if (active) {
    const auto start = [&](int i) { return hash_unit(((uint64_t)P.g_off << 20) ^ ((uint64_t)j << 32) ^ (uint64_t)i); };
    il_factor(d, e, n, lam[j], tiny, start, y, wb + nc + t, wb + 2 * nc + t, zb + t, cnt);
    for (int it = 0; it < INV_ITERS; ++it) {
      if (it > 0) il_forward(n, inv, y, zb + t, cnt);
      inv = 1.0 / sqrt(il_back(e, n, y, wb + nc + t, wb + 2 * nc + t, zb + t, cnt));
    }
  }
  __syncthreads();  // every thread's multipliers in Z are dead
  if (active) {
    double* z = zb + (int64_t)n * t;
    int i = 0;
    for (; i + PF <= n; i += PF) {
      double v[PF];
#pragma unroll
      for (int k = 0; k < PF; ++k) v[k] = y[(int64_t)(i + k) * cnt];
#pragma unroll
      for (int k = 0; k < PF; ++k) z[i + k] = v[k] * inv;
    }
    for (; i < n; ++i) z[i] = y[(int64_t)i * cnt] * inv;
  }
  // launched alongside eigvecs_small: complete only when that is
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// (2a) Gram matrix, lower 64 x 64 tiles (a >= b): G[r + m c] = sum_i Z[i, r] Z[i, c],
// G at work + 3 g_off, leading dimension m = nvec.  On the FP64 tensor path, the
// fragments straight from Z (four rows of a column are a 32-byte sector): a warp has
// a 32 x 32 quadrant for every other group of 8 rows.  At bond dimension 3072
// 342 -> 162 us (16-row stages through shared memory, on the FP64 pipe).
__global__ void __launch_bounds__(256)
gram_tiles(const EigDev* __restrict__ probs, const TileTask* __restrict__ tasks, const double* Zg, double* work,
           const int* __restrict__ flags) {
  __shared__ double half[4][32][33];
  const TileTask tk = tasks[blockIdx.x];
  if (flags[tk.prob]) return;
  const EigDev P = probs[tk.prob];
  const int n = P.n, m = P.nvec;
  const double* Z = Zg + P.g_off;
  double* Gm = work + 3 * P.g_off;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  const int r0 = tk.a * GT + 32 * (warp & 1), c0 = tk.b * GT + 32 * ((warp >> 1) & 1), kh = warp >> 2;
  double acc[4][4][2] = {};
  const double *za[4], *zb[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {  // columns past the last repeat it; they are not stored
    za[q] = Z + (int64_t)n * min(r0 + 8 * q + g, m - 1) + t4;
    zb[q] = Z + (int64_t)n * min(c0 + 8 * q + g, m - 1) + t4;
  }
  auto load = [&](int i, double (&a)[2][4], double (&b)[2][4]) {
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool in = i + 4 * s + t4 < n;
        a[s][q] = in ? za[q][i + 4 * s] : 0.0;
        b[s][q] = in ? zb[q][i + 4 * s] : 0.0;
      }
  };
  auto use = [&](const double (&a)[2][4], const double (&b)[2][4]) {
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w) dmma_tr(acc[u][w], a[s][u], b[s][w]);
  };
  double a0[2][4], b0[2][4], a1[2][4], b1[2][4];
  load(8 * kh, a0, b0);
  for (int i = 8 * kh; i < n; i += 32) {  // one group in flight while the other is used
    load(i + 16, a1, b1);
    use(a0, b0);
    load(i + 32, a0, b0);
    use(a1, b1);
  }
  if (kh == 1) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int w = 0; w < 4; ++w)
#pragma unroll
        for (int x = 0; x < 2; ++x) half[warp & 3][8 * u + g][8 * w + 2 * t4 + x] = acc[u][w][x];
  }
  __syncthreads();
  if (kh == 1) return;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int w = 0; w < 4; ++w)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int r = r0 + 8 * u + g, c = c0 + 8 * w + 2 * t4 + x;
        if (r < m && c < m && r >= c) Gm[r + (int64_t)m * c] = acc[u][w][x] + half[warp][8 * u + g][8 * w + 2 * t4 + x];
      }
}

// The triangular solve both (2b) and (2c) need, one row per thread:
// x <- x L^-T for the 32 x 32 lower triangle whose column c is lt[c][.], rd its
// reciprocal diagonal.  Column by column, so that the chain is one product and one
// sum each; two entries of L per load, the same for every thread of the warp.
__device__ __forceinline__ void solve_row(double (&x)[CH_PB], const double (*lt)[CH_LD], const double* rd) {
#pragma unroll
  for (int c = 0; c < CH_PB; ++c) {
    x[c] *= rd[c];
#pragma unroll
    for (int q = (c + 1) / 2; q < CH_PB / 2; ++q) {
      const double2 l = *reinterpret_cast<const double2*>(&lt[c][2 * q]);
      if (2 * q > c) x[2 * q] = fma(-x[c], l.x, x[2 * q]);
      x[2 * q + 1] = fma(-x[c], l.y, x[2 * q + 1]);
    }
  }
}

// (2b) Cholesky G = L L^T of the lower triangle in place, right-looking with
// 32-column panels, one cluster per problem.  Every CTA factors the diagonal block
// for itself (a warp with a row per lane), then the panel's rows go to the cluster's
// warps 32 at a time, then the trailing matrix 32 x 32 at a time on the FP64 tensor
// path, the fragments straight from L2, all loads of a tile in flight (two k steps
// at a time by twice the warps: 646 us).  A panel is a chain of L2 latencies and two
// cluster barriers.  At bond dimension 3072 1221 -> 372 us (three barriers per
// column of the block, divisions, 64 x 64 tiles on the FP64 pipe).  Pivots below
// COLLAPSE_PIVOT2 (first pass) flag the problem; a flagged or non-positive pivot is
// replaced by 1 so the arithmetic stays finite (the problem is redone by the fallback).
__global__ void __launch_bounds__(CH_THREADS)
chol_cluster(const EigDev* __restrict__ probs, double* work, int* flags, int check) {
  __shared__ __align__(16) double lt[CH_PB][CH_LD];
  __shared__ double rd[CH_PB];
  cgx::cluster_group cluster = cgx::this_cluster();
  const int CL = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int pi = blockIdx.x / CL;
  const bool redo = flags[pi] != 0;
  cluster.sync();  // read by every CTA before CTA 0 may raise it: the whole cluster goes on or returns
  if (redo) return;
  const EigDev P = probs[pi];
  const int m = P.nvec;
  double* A = work + 3 * P.g_off;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int unit0 = rank + CL * warp, units = CL * (CH_THREADS / 32);  // this warp's place in the cluster
  for (int p0 = 0; p0 < m; p0 += CH_PB) {
    const int pb = min(CH_PB, m - p0);
    // (i) the diagonal block, lane r its row r; the unit matrix past the last row
    if (warp == 0) {
      double a[CH_PB];
#pragma unroll
      for (int c = 0; c < CH_PB; ++c)
        a[c] = lane < pb && c <= lane ? A[(p0 + lane) + (int64_t)m * (p0 + c)] : (c == lane ? 1.0 : 0.0);
      bool bad = false;
      double my_rd = 1.0;
#pragma unroll
      for (int k = 0; k < CH_PB; ++k) {
        double piv = __shfl_sync(0xffffffffu, a[k], k);
        if (!(piv > (check ? COLLAPSE_PIVOT2 : 0.0)) && k < pb) {
          bad = true;
          piv = 1.0;
        }
        const double ri = rsqrt(piv);
        if (lane == k) my_rd = ri;
        a[k] = lane == k ? piv * ri : (lane > k ? a[k] * ri : 0.0);
        lt[k][lane] = a[k];
        __syncwarp();
#pragma unroll
        for (int q = (k + 1) / 2; q < CH_PB / 2; ++q) {
          const double2 l = *reinterpret_cast<const double2*>(&lt[k][2 * q]);
          if (2 * q > k) a[2 * q] = fma(-a[k], l.x, a[2 * q]);
          a[2 * q + 1] = fma(-a[k], l.y, a[2 * q + 1]);
        }
      }
      rd[lane] = my_rd;
      if (rank == 0 && bad && lane == 0 && atomicExch(&flags[pi], 1) == 0) atomicAdd(&g_eig_redo, 1ull);
    }
    __syncthreads();
    // (ii) rows below the block: L[i, p0:p0+pb] = A[i, p0:p0+pb] L_pp^-T
    const int rbeg = p0 + pb;  // pb < 32 in the last panel only, which has none
    for (int i = rbeg + 32 * unit0 + lane; i < m; i += 32 * units) {
      double x[CH_PB];
#pragma unroll
      for (int k = 0; k < CH_PB; ++k) x[k] = A[i + (int64_t)m * (p0 + k)];
      asm volatile("" : : : "memory");  // or the triangle is kept over the loop, in local memory
      solve_row(x, lt, rd);
#pragma unroll
      for (int k = 0; k < CH_PB; ++k) A[i + (int64_t)m * (p0 + k)] = x[k];
    }
    __threadfence();
    cluster.sync();
    if (rank == 0 && warp == 0)  // every CTA has read the block
#pragma unroll
      for (int c = 0; c < CH_PB; ++c)
        if (lane < pb && c <= lane) A[(p0 + lane) + (int64_t)m * (p0 + c)] = lt[c][lane];
    if (rbeg >= m) break;
    // (iii) trailing update of the lower tiles (ta >= tb) of A[rbeg:, rbeg:]
    const int nt = (m - rbeg + 31) >> 5, ntiles = nt * (nt + 1) / 2;
    const int g = lane >> 2, t4 = lane & 3;
    for (int t = unit0; t < ntiles; t += units) {
      int ta = 0;
      while ((ta + 1) * (ta + 2) / 2 <= t) ++ta;
      const int tb = t - ta * (ta + 1) / 2;
      const int ra = rbeg + 32 * ta, rb = rbeg + 32 * tb;
      const double *la[4], *lb[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // rows past the last repeat it; they are not stored
        la[q] = A + min(ra + 8 * q + g, m - 1) + (int64_t)m * (p0 + t4);
        lb[q] = A + min(rb + 8 * q + g, m - 1) + (int64_t)m * (p0 + t4);
      }
      double acc[4][4][2], a[CH_PB / 4][4], b[CH_PB / 4][4];  // all loads in flight at once
#pragma unroll
      for (int k = 0; k < CH_PB / 4; ++k)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a[k][q] = -la[q][(int64_t)m * (4 * k)];
          b[k][q] = lb[q][(int64_t)m * (4 * k)];
        }
      auto own = [&](int r, int c) { return r < m && c <= r; };
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int r = ra + 8 * u + g, c = rb + 8 * w + 2 * t4 + x;
            acc[u][w][x] = own(r, c) ? A[r + (int64_t)m * c] : 0.0;
          }
#pragma unroll
      for (int k = 0; k < CH_PB / 4; ++k)
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int w = 0; w < 4; ++w) dmma_tr(acc[u][w], a[k][u], b[k][w]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int r = ra + 8 * u + g, c = rb + 8 * w + 2 * t4 + x;
            if (own(r, c)) A[r + (int64_t)m * c] = acc[u][w][x];
          }
    }
    __threadfence();
    cluster.sync();
  }
}

// (2c) Z <- Z L^-T, row by row (rows are independent): TS_ROWS rows per CTA, columns
// in 32-wide panels.  The solved part enters through 32 x 32 products on the FP64
// tensor path, a warp per 32 solved columns, the fragments straight from L2 and L1,
// all loads of a product in flight; the panel's own triangle by substitution.  At
// bond dimension 3072 693 -> 312 us; with eight warps of 128 registers and part of
// the loads in flight 390 to 490.
__global__ void __launch_bounds__(TS_THREADS, 2)
trsm_rows(const EigDev* __restrict__ probs, const VecTask* __restrict__ tasks, double* Zg, const double* work,
          const int* __restrict__ flags) {
  __shared__ double zx[TS_ROWS][CH_PB + 1];  // the panel's columns of the rows
  __shared__ __align__(16) double lt[CH_PB][CH_LD];
  __shared__ double rd[CH_PB];
  const VecTask tk = tasks[blockIdx.x];
  if (flags[tk.prob]) return;
  const EigDev P = probs[tk.prob];
  const int n = P.n, m = P.nvec;
  double* Z = Zg + P.g_off;
  const double* L = work + 3 * P.g_off;
  const int i0 = tk.j0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  for (int p0 = 0; p0 < m; p0 += CH_PB) {
    const int pb = min(CH_PB, m - p0);
    __syncthreads();  // the columns solved before are complete; zx and lt are free
    for (int e2 = tid; e2 < TS_ROWS * CH_PB; e2 += TS_THREADS) {
      const int r = e2 % TS_ROWS, c = e2 / TS_ROWS;
      zx[r][c] = i0 + r < n && c < pb ? Z[(i0 + r) + (int64_t)n * (p0 + c)] : 0.0;
      const double l = r < pb && c <= r ? L[(p0 + r) + (int64_t)m * (p0 + c)] : 0.0;
      lt[c][r] = l;
      if (r == c) rd[c] = c < pb ? 1.0 / l : 0.0;
    }
    double acc[4][4][2] = {};
    const bool busy = 32 * warp < p0;
    if (busy) {
      const double *xa[4], *lb[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // rows past the last repeat it; they are not stored
        xa[q] = Z + min(i0 + 8 * q + g, n - 1) + (int64_t)n * t4;
        lb[q] = L + min(p0 + 8 * q + g, m - 1) + (int64_t)m * t4;
      }
      for (int k0 = 32 * warp; k0 < p0; k0 += TS_THREADS) {
        double a[CH_PB / 4][4], b[CH_PB / 4][4];  // all loads in flight at once
#pragma unroll
        for (int k = 0; k < CH_PB / 4; ++k)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            a[k][q] = xa[q][(int64_t)n * (k0 + 4 * k)];
            b[k][q] = lb[q][(int64_t)m * (k0 + 4 * k)];
          }
#pragma unroll
        for (int k = 0; k < CH_PB / 4; ++k)
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int w = 0; w < 4; ++w) dmma_tr(acc[u][w], a[k][u], b[k][w]);
      }
    }
    __syncthreads();
    for (int q = 0; q < TS_THREADS / 32 && 32 * q < p0; ++q) {  // one warp after the other: the same order always
      if (warp == q) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int w = 0; w < 4; ++w)
#pragma unroll
            for (int x = 0; x < 2; ++x) zx[8 * u + g][8 * w + 2 * t4 + x] -= acc[u][w][x];
      }
      __syncthreads();
    }
    if (warp == 0) {
      double x[CH_PB];
#pragma unroll
      for (int c = 0; c < CH_PB; ++c) x[c] = zx[lane][c];
      solve_row(x, lt, rd);
      if (i0 + lane < n) {
#pragma unroll
        for (int c = 0; c < CH_PB; ++c)
          if (c < pb) Z[(i0 + lane) + (int64_t)n * (p0 + c)] = x[c];
      }
    }
  }
}

// entry (row i, reflector a) of the panel of mm reflectors from k0 on: the kept part
// of column k0 + a below the subdiagonal, 1 on it, 0 above and past the ends
__device__ __forceinline__ double reflector_entry(const double* Gp, int n, int k0, int mm, int i, int a) {
  const int ka = k0 + a;
  if (a >= mm || i >= n || i <= ka) return 0.0;
  return i == ka + 1 ? 1.0 : Gp[i + (int64_t)n * ka];
}

// (3a) compact-WY factor T of the reflectors [32 b, 32 b + 32) of a problem:
// S = V^T V (v_k(k+1) = 1, v_k(i) = G(i, k) for i >= k + 2), then the dlarft
// recurrence T(0:c, c) = -tau_c T(0:c, 0:c) S(0:c, c), T(c, c) = tau_c
__global__ void __launch_bounds__(256)
wy_factors(const EigDev* __restrict__ probs, const TileTask* __restrict__ tasks, const double* G, const double* Tg,
           double* work, const int* __restrict__ flags) {
  __shared__ double S[BT_NB][BT_NB + 1];
  __shared__ double T[BT_NB][BT_NB + 1];
  const TileTask tk = tasks[blockIdx.x];
  if (flags[tk.prob]) return;
  const EigDev P = probs[tk.prob];
  const int n = P.n;
  const double* Gp = G + P.g_off;
  const double* tau = Tg + 3 * P.w_off + 2 * n;
  const int k0 = tk.a * BT_NB, mm = min(BT_NB, n - 2 - k0);
  double* Tout = work + 3 * P.g_off + (int64_t)P.nvec * P.nvec + (int64_t)tk.a * BT_NB * BT_NB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  // on the FP64 tensor path: a warp takes every eighth group of 8 rows, and one
  // fragment of V serves on both sides (at bond dimension 3072 425 -> 43 us; a warp
  // per dot product read each reflector 31 times)
  double acc[4][4][2] = {};
  for (int i = k0 + 1 + 8 * warp; i < n; i += 128) {
    double v[2][2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          v[u][x][q] = reflector_entry(Gp, n, k0, mm, i + 64 * u + 4 * x + t4, 8 * q + g);
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int c = 0; c < 4; ++c) dmma_tr(acc[a][c], v[u][x][a], v[u][x][c]);
  }
  for (int q = 0; q < 8; ++q) {
    if (warp == q) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            double& s = S[8 * a + g][8 * c + 2 * t4 + x];
            s = q == 0 ? acc[a][c][x] : s + acc[a][c][x];
          }
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) {
    for (int c = 0; c < mm; ++c) {
      const double tc = tau[k0 + c];
      // T(a, c) = -tc * sum_{b in [a, c)} T(a, b) S(b, c), lanes over a
      double x = 0.0;
      if (lane < c) {
        for (int b = lane; b < c; ++b) x += T[lane][b] * S[b][c];
        T[lane][c] = -tc * x;
      }
      if (lane == 0) T[c][c] = tc;
      __syncwarp();
    }
  }
  __syncthreads();
  for (int e2 = threadIdx.x; e2 < BT_NB * BT_NB; e2 += blockDim.x) {
    const int a = e2 % BT_NB, c = e2 / BT_NB;
    Tout[e2] = (a < mm && c < mm && a <= c) ? T[a][c] : 0.0;
  }
}

// (3b) z = Q y for the vectors [j0, j0 + BT_VB) of a problem: panels last to
// first, Y <- Y - V (T (V^T Y)) over rows >= k0 + 1; then the gauge (largest
// magnitude entry positive, first on ties).  All three products are on the FP64
// tensor path, with the fragments of V and Y straight from L2: 16 warps with some
// 24 loads each in flight, and no barrier inside a product.  At bond dimension 3072
// 2390 -> 890 us (64-row stages through shared memory, on the FP64 pipe); V comes
// from L2 twice.
__global__ void __launch_bounds__(512)
wy_apply(const EigDev* __restrict__ probs, const VecTask* __restrict__ tasks, const double* G, double* Zg,
         const double* work, const int* __restrict__ flags) {
  constexpr int XLD = BT_VB + 4;  // a fragment's rows on different banks
  __shared__ double part[4][BT_NB][BT_VB];
  __shared__ double X[BT_NB][XLD], X2[BT_NB][XLD];
  const VecTask tk = tasks[blockIdx.x];
  if (flags[tk.prob]) return;
  const EigDev P = probs[tk.prob];
  const int n = P.n, nv = min(BT_VB, P.nvec - tk.j0);
  const double* Gp = G + P.g_off;
  double* Y = Zg + P.g_off + (int64_t)n * tk.j0;
  const double* Tst = work + 3 * P.g_off + (int64_t)P.nvec * P.nvec;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int npan = (n - 2 + BT_NB - 1) / BT_NB;
  for (int pnl = npan - 1; pnl >= 0; --pnl) {
    const int k0 = pnl * BT_NB, mm = min(BT_NB, n - 2 - k0);
    __syncthreads();  // Y of the panel before is complete
    // X = V^T Y over rows >= k0 + 1, a warp every 16th group of 8 rows
    {
      double acc[4][2][2] = {};
      for (int i = k0 + 1 + 8 * warp; i < n; i += 256) {
        double v[2][2][4], y[2][2][2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int r = i + 128 * u + 4 * x + t4;
#pragma unroll
            for (int q = 0; q < 4; ++q) v[u][x][q] = reflector_entry(Gp, n, k0, mm, r, 8 * q + g);
#pragma unroll
            for (int q = 0; q < 2; ++q) y[u][x][q] = r < n && 8 * q + g < nv ? Y[r + (int64_t)n * (8 * q + g)] : 0.0;
          }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
              for (int c = 0; c < 2; ++c) dmma_tr(acc[a][c], v[u][x][a], y[u][x][c]);
      }
      for (int q = 0; q < 4; ++q) {  // four warps at a time, in order
        if (warp >> 2 == q) {
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                double& s = part[warp & 3][8 * a + g][8 * c + 2 * t4 + x];
                s = q == 0 ? acc[a][c][x] : s + acc[a][c][x];
              }
        }
        __syncthreads();
      }
      const int a = tid / BT_VB, c = tid % BT_VB;
      X[a][c] = (part[0][a][c] + part[1][a][c]) + (part[2][a][c] + part[3][a][c]);
    }
    __syncthreads();
    // X2 = T X (T upper triangular), an 8 x 8 tile per warp
    if (warp < 8) {
      const int a = 8 * (warp >> 1), c = 8 * (warp & 1);
      double tf[8], acc[2] = {};
#pragma unroll
      for (int k = 0; k < 8; ++k) tf[k] = Tst[(int64_t)pnl * BT_NB * BT_NB + a + g + BT_NB * (4 * k + t4)];
#pragma unroll
      for (int k = 0; k < 8; ++k) dmma_tr(acc, tf[k], X[4 * k + t4][c + g]);
      X2[a + g][c + 2 * t4] = acc[0];
      X2[a + g][c + 2 * t4 + 1] = acc[1];
    }
    __syncthreads();
    // Y -= V X2
    double xf[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int c = 0; c < 2; ++c) xf[k][c] = X2[4 * k + t4][8 * c + g];
    for (int i = k0 + 1 + 8 * warp; i < n; i += 256) {
      double v[2][8], y[2][2][2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = i + 128 * u + g;
#pragma unroll
        for (int k = 0; k < 8; ++k) v[u][k] = -reflector_entry(Gp, n, k0, mm, r, 4 * k + t4);
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int col = 8 * c + 2 * t4 + x;
            y[u][c][x] = r < n && col < nv ? Y[r + (int64_t)n * col] : 0.0;
          }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = i + 128 * u + g;
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int c = 0; c < 2; ++c) dmma_tr(y[u][c], v[u][k], xf[k][c]);
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int col = 8 * c + 2 * t4 + x;
            if (r < n && col < nv) Y[r + (int64_t)n * col] = y[u][c][x];
          }
      }
    }
  }
  __syncthreads();
  // gauge, one warp per vector
  if (warp < nv) {
    double* y = Y + (int64_t)n * warp;
    double best = -1.0;
    int bi = n;
    for (int i = lane; i < n; i += 32) {
      const double a = fabs(y[i]);
      if (a > best) { best = a; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    const bool flip = bi < n && y[bi] < 0.0;
    __syncwarp();
    if (flip)
      for (int i = lane; i < n; i += 32) y[i] = -y[i];
  }
}

std::vector<EigDev> to_dev(const tt_eig_problem* probs, int n_probs, const int* nvec) {
  std::vector<EigDev> hp(n_probs);
  for (int i = 0; i < n_probs; ++i)
    hp[i] = EigDev{probs[i].g_off, probs[i].w_off, probs[i].a_off, probs[i].n, probs[i].flags,
                   nvec ? nvec[i] : 0, 0, 0};
  return hp;
}

constexpr int64_t kVecsSmemCap = 28 * 1024;  // doubles (224 KB) of dynamic shared memory of eigvecs_small

// Sectors above the size of the one-CTA kernels go to the cluster kernels.
bool is_big(const EigDev& e) { return e.n > SN && !(e.flags & TT_EIG_ROW_1X2); }

// The cluster reduction for sectors of up to n states
const void* vals_kernel(int n) {
  return n <= 2 * CR_THREADS   ? (const void*)tridiag_eigvals_cluster<2>
         : n <= 4 * CR_THREADS ? (const void*)tridiag_eigvals_cluster<4>
                               : (const void*)tridiag_eigvals_cluster<8>;
}
constexpr int CR_MAX = 8 * CR_THREADS;  // states of a sector that it takes, at most

// Whether a batch of cluster-sized sectors goes to the blocked reduction: its largest
// has more states than the other takes, or is one of those (1800 up) for which both
// triangles of all sectors together must stay in L2.
bool blocked_sectors(const std::vector<EigDev>& big) {
  int n = 0;
  int64_t bytes = 0;
  for (const EigDev& e : big) {
    n = std::max(n, e.n);
    bytes += (int64_t)sizeof(double) * e.n * e.n;
  }
  return n > CR_MAX || (n > 1800 && bytes > 100000000);
}

// Cluster size and shared-memory caps of the cluster kernels on this thread's
// device: 16 CTAs per cluster when the device can co-schedule that many with
// the full shared-memory carve-out, else 8, else none (an error for sectors that
// need them).
struct ClusterPlan {
  int device = -1;
  int cl = 0;
  int64_t vals_cap = 0, blocked_cap = 0, vecs_cap = 0;  // doubles of dynamic shared memory per CTA
};

const ClusterPlan& cluster_plan(tt_ctx* ctx) {
  static thread_local ClusterPlan cp;
  if (cp.device == ctx->device) return cp;
  cp = ClusterPlan();
  cp.device = ctx->device;
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess) {
    cudaGetLastError();
    return cp;
  }
  constexpr int NK = 5;
  const void* kernels[NK] = {vals_kernel(1), vals_kernel(4 * CR_THREADS), vals_kernel(CR_MAX),
                             (const void*)tridiag_blocked_cluster, (const void*)tridiag_eigvecs_cluster};
  int64_t caps[NK];
  for (int k = 0; k < NK; ++k) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kernels[k]) != cudaSuccess) {
      cudaGetLastError();
      return cp;
    }
    caps[k] = ((int64_t)optin - (int64_t)fa.sharedSizeBytes - 1024) / 8;
  }
  const int64_t va = std::min({caps[0], caps[1], caps[2]}), vc = caps[3], vb = caps[4];
  if (vb < 6 * MAX_N) return cp;
  for (int k = 0; k < NK; ++k) {
    if (cudaFuncSetAttribute(kernels[k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(caps[k] * 8)) !=
            cudaSuccess ||
        cudaFuncSetAttribute(kernels[k], cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      return cp;
    }
  }
  if (cudaFuncSetAttribute(chol_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return cp;
  }
  for (int cl : {CL_MAX, 8}) {
    // the largest sectors fit, the blocked reduction's at the narrowest panel
    bool ok = cluster_layout(CR_MAX, cl, va).nb > 0 && blocked_smem(MAX_N, 8, cl) <= vc;
    for (int k = 0; k < NK && ok; ++k) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = cl;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(cl);
      cfg.blockDim = dim3(k < 3 ? CR_THREADS : TT);
      cfg.dynamicSmemBytes = (size_t)(caps[k] * 8);
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int nc = 0;
      if (cudaOccupancyMaxActiveClusters(&nc, kernels[k], &cfg) != cudaSuccess) {
        cudaGetLastError();
        nc = 0;
      }
      ok = nc >= 1;
    }
    if (ok) {
      cp.cl = cl;
      break;
    }
  }
  cp.vals_cap = va;
  cp.blocked_cap = vc;
  cp.vecs_cap = vb;
  return cp;
}

// A launch in clusters of `cl` CTAs (0: none) with `smem` bytes of dynamic
// shared memory.  With `beside` it may start while the launch before it still
// runs (that one says so, and this one ends with a wait for it).
template <class... Args>
cudaError_t launch(tt_ctx* ctx, int grid, int block, int cl, size_t smem, bool beside, const void* kernel,
                   Args... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  unsigned na = 0;
  if (cl > 0) {
    at[na].id = cudaLaunchAttributeClusterDimension;
    at[na].val.clusterDim.x = cl;
    at[na].val.clusterDim.y = 1;
    at[na++].val.clusterDim.z = 1;
  }
  if (beside) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = na;
  void* argv[] = {(void*)&args...};
  const cudaError_t e = cudaLaunchKernelExC(&cfg, kernel, argv);
  tt::count_launch(ctx);
  return e;
}

// One cluster of `cl` CTAs per problem; `need` doubles of dynamic shared memory.
template <class... Args>
cudaError_t launch_cluster(tt_ctx* ctx, int cl, int threads, int n_probs, int64_t need, const void* kernel, Args... args) {
  return launch(ctx, cl * n_probs, threads, cl, (size_t)(need * 8), false, kernel, args...);
}

}  // namespace

extern "C" {

int tt_sym_eigvals_batched(tt_ctx* ctx, const tt_eig_problem* probs, int n_probs, double* G, double* T,
                           double* w, const double* A) {
  TT_REQUIRE(ctx && (n_probs == 0 || (probs && G && T && w)), "tt_sym_eigvals_batched: null argument");
  if (n_probs == 0) return TT_OK;
  for (int i = 0; i < n_probs; ++i) {
    TT_REQUIRE(probs[i].n >= 0 && probs[i].n <= MAX_N, "tt_sym_eigvals_batched: n must be 0..4096");
    if (probs[i].flags & TT_EIG_ROW_1X2)
      TT_REQUIRE(probs[i].n == 2 && A, "tt_sym_eigvals_batched: 1x2 case needs n == 2 and A");
  }
  std::vector<EigDev> all = to_dev(probs, n_probs, nullptr);
  const ClusterPlan& cp = cluster_plan(ctx);
  std::vector<EigDev> hp, big;  // small problems first, then the cluster ones
  int nsmall_max = 1;
  for (const EigDev& e : all) {
    (is_big(e) ? big : hp).push_back(e);
    if (!is_big(e)) nsmall_max = std::max(nsmall_max, e.n);
  }
  const int n_small = (int)hp.size();
  int64_t need = 0, scratch = 0;
  int nbig_max = 0;
  const bool blocked = blocked_sectors(big);
  int cl = cp.cl;
  if (!big.empty()) {
    TT_REQUIRE(cp.cl > 0, "tt_sym_eigvals_batched: no thread-block clusters for sectors of this size");
    for (const EigDev& e : big) nbig_max = std::max(nbig_max, e.n);
    // More clusters than run at once: smaller ones, as long as their CTAs hold the
    // columns in shared memory.  In clusters of 16, 20 sectors of 130 took 1291 us and
    // 100 of 160 7.73 ms (one CTA each, before: 937 us and 1.35 ms), so 469 us and 1.48
    // ms; 74 of 220 8.0 -> 2.6 ms, 36 of 260 5.3 -> 2.2.
    while (!blocked && cl > 2 && (int64_t)big.size() * cl > ctx->num_sms &&
           cluster_layout(nbig_max, cl / 2, cp.vals_cap).resident)
      cl /= 2;
    for (EigDev& e : big) {
      if (blocked) {  // the widest panel whose shared memory fits
        e.nb = PNB_MAX;
        while (e.nb > 8 && blocked_smem(e.n, e.nb, cp.cl) > cp.blocked_cap) e.nb /= 2;
        need = std::max(need, blocked_smem(e.n, e.nb, cp.cl));
        TT_REQUIRE(need <= cp.blocked_cap, "tt_sym_eigvals_batched: sector too large for the cluster eigensolver");
        e.s_off = scratch;
        scratch += (int64_t)e.n * 2 * e.nb;
        continue;
      }
      const ClusterLayout L = cluster_layout(e.n, cl, cp.vals_cap);
      TT_REQUIRE(L.nb > 0, "tt_sym_eigvals_batched: sector too large for the cluster eigensolver");
      // the layouts of later stages take what there is
      need = std::max(need, L.resident ? L.doubles : cp.vals_cap);
      e.s_off = scratch;
      scratch += (int64_t)cl * ((e.n + cl - 1) / cl) * cl_ld(e.n);
    }
  }
  hp.insert(hp.end(), big.begin(), big.end());
  // every sector's eigenvalues, BS_PER per CTA over the whole GPU
  std::vector<VecTaskB> bt;
  int nmax = 1;
  for (int p = 0; p < (int)hp.size(); ++p) {
    if (hp[p].flags & TT_EIG_ROW_1X2) continue;
    nmax = std::max(nmax, hp[p].n);
    for (int j0 = 0; j0 < hp[p].n; j0 += BS_PER) bt.push_back(VecTaskB{p, j0});
  }
  // problems, bisection tasks and the reductions' scratch in one buffer
  const size_t pb = sizeof(EigDev) * hp.size(), tb = (sizeof(VecTaskB) * bt.size() + 15) & ~(size_t)15;
  std::vector<char> host(pb + tb);
  std::memcpy(host.data(), hp.data(), pb);
  if (!bt.empty()) std::memcpy(host.data() + pb, bt.data(), sizeof(VecTaskB) * bt.size());
  char* buf = tt::pool_alloc<char>(ctx, pb + tb + sizeof(double) * (size_t)scratch);
  if (!buf) return tt::fail(TT_ERR_OOM, "tt_sym_eigvals_batched: allocation failed");
  TT_CUDA(tt::h2d_async(ctx, buf, host.data(), host.size()));
  const EigDev* dp = reinterpret_cast<const EigDev*>(buf);
  const VecTaskB* d_bt = reinterpret_cast<const VecTaskB*>(buf + pb);
  double* sc = reinterpret_cast<double*>(buf + pb + tb);
  static thread_local uint64_t attr = 0;  // per host thread and device
  if (tt::first_on_device(attr, ctx->device)) {
    TT_CUDA(cudaFuncSetAttribute(tridiag_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * small_smem(SN, TT / 32))));
    TT_CUDA(cudaFuncSetAttribute(bisect_sectors, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double2) * MAX_N)));
  }
  if (n_small > 0) {
    const int threads = small_threads(nsmall_max);
    tridiag_small<<<n_small, threads, sizeof(double) * (size_t)small_smem(nsmall_max, threads / 32), ctx->stream>>>(
        dp, G, T, w, A);
    TT_LAUNCH_CHECK(ctx);
  }
  if (blocked) {
    TT_CUDA(launch_cluster(ctx, cp.cl, TT, (int)big.size(), need, (const void*)tridiag_blocked_cluster, dp + n_small, G,
                           T, sc));
  } else if (!big.empty()) {
    TT_CUDA(launch(ctx, cl * (int)big.size(), CR_THREADS, cl, (size_t)(need * 8), n_small > 0,
                   vals_kernel(nbig_max), dp + n_small, G, T, sc, need));
  }
  if (!bt.empty()) {
    const size_t bs_smem = sizeof(double2) * (size_t)((nmax + 7) & ~7);
    bisect_sectors<<<(unsigned)bt.size(), BS_THREADS, bs_smem, ctx->stream>>>(dp, d_bt, T, w);
    TT_LAUNCH_CHECK(ctx);
  }
  tt::pool_free(ctx, buf);
  return TT_OK;
}

int tt_eig_redo_count(tt_ctx* ctx, int64_t* count) {
  TT_REQUIRE(ctx && count, "tt_eig_redo_count: null argument");
  unsigned long long* h = reinterpret_cast<unsigned long long*>(ctx->h_scalars);
  TT_CUDA(cudaMemcpyFromSymbolAsync(h, g_eig_redo, sizeof(unsigned long long), 0, cudaMemcpyDeviceToHost,
                                    ctx->stream));
  TT_CUDA(cudaStreamSynchronize(ctx->stream));
  *count = (int64_t)*h;
  return TT_OK;
}

int tt_sym_eigvecs_batched(tt_ctx* ctx, const tt_eig_problem* probs, int n_probs, const int* nvec,
                           const double* G, const double* T, const double* w, double* Z, double* work,
                           const double* A) {
  TT_REQUIRE(ctx && (n_probs == 0 || (probs && nvec && G && T && w && Z && work)),
             "tt_sym_eigvecs_batched: null argument");
  if (n_probs == 0) return TT_OK;
  for (int i = 0; i < n_probs; ++i) {
    TT_REQUIRE(probs[i].n >= 0 && probs[i].n <= MAX_N, "tt_sym_eigvecs_batched: n must be 0..4096");
    TT_REQUIRE(nvec[i] >= 0 && nvec[i] <= probs[i].n && nvec[i] <= MAX_N / 2,
               "tt_sym_eigvecs_batched: nvec must be 0..min(n, 2048)");
    if (probs[i].flags & TT_EIG_ROW_1X2) TT_REQUIRE(A, "tt_sym_eigvecs_batched: 1x2 case needs A");
  }
  std::vector<EigDev> all = to_dev(probs, n_probs, nvec);
  const ClusterPlan& cp = cluster_plan(ctx);
  std::vector<EigDev> hp, big;  // small problems first, then the cluster ones
  int nsmall_max = 1;
  for (const EigDev& e : all) {
    (is_big(e) ? big : hp).push_back(e);
    if (!is_big(e)) nsmall_max = std::max(nsmall_max, e.n);
  }
  TT_REQUIRE(big.empty() || cp.cl > 0, "tt_sym_eigvecs_batched: no thread-block clusters for sectors of this size");
  const int n_small = (int)hp.size(), nbig = (int)big.size();
  int nbig_max = 0;
  for (const EigDev& e : big) nbig_max = std::max(nbig_max, e.n);
  hp.insert(hp.end(), big.begin(), big.end());
  std::vector<VecTask> iv, ts, ap;
  std::vector<TileTask> gm, wy;
  for (int p = 0; p < nbig; ++p) {
    const EigDev& e = big[p];
    for (int j = 0; j < e.nvec; j += IV_THREADS) iv.push_back(VecTask{p, j});
    const int nt = (e.nvec + GT - 1) / GT;
    for (int a = 0; a < nt; ++a)
      for (int b = 0; b <= a; ++b) gm.push_back(TileTask{p, a, b});
    if (e.nvec > 0) {
      for (int i = 0; i < e.n; i += TS_ROWS) ts.push_back(VecTask{p, i});
      for (int k = 0; k * BT_NB < e.n - 2; ++k) wy.push_back(TileTask{p, k, 0});
      for (int j = 0; j < e.nvec; j += BT_VB) ap.push_back(VecTask{p, j});
    }
  }
  // problems, task lists and the (zero) flags in one buffer, one copy
  std::vector<char> host;
  auto put = [&](const auto& v) {
    const size_t at = host.size();
    host.resize((at + v.size() * sizeof(v[0]) + 15) & ~(size_t)15);
    if (!v.empty()) std::memcpy(host.data() + at, v.data(), v.size() * sizeof(v[0]));
    return at;
  };
  put(hp);
  const size_t at_iv = put(iv), at_ts = put(ts), at_ap = put(ap), at_gm = put(gm), at_wy = put(wy);
  const size_t at_flags = put(std::vector<int>((size_t)nbig + 1, 0));
  char* buf = tt::pool_alloc<char>(ctx, host.size());
  if (!buf) return tt::fail(TT_ERR_OOM, "tt_sym_eigvecs_batched: allocation failed");
  TT_CUDA(tt::h2d_async(ctx, buf, host.data(), host.size()));
  const EigDev* dp = reinterpret_cast<const EigDev*>(buf);
  const EigDev* db = dp + n_small;
  const VecTask* d_iv = reinterpret_cast<const VecTask*>(buf + at_iv);
  const VecTask* d_ts = reinterpret_cast<const VecTask*>(buf + at_ts);
  const VecTask* d_ap = reinterpret_cast<const VecTask*>(buf + at_ap);
  const TileTask* d_gm = reinterpret_cast<const TileTask*>(buf + at_gm);
  const TileTask* d_wy = reinterpret_cast<const TileTask*>(buf + at_wy);
  int* flags = reinterpret_cast<int*>(buf + at_flags);
  // shared memory for the largest problem whose factors fit, or its vectors alone
  int64_t need = 0;
  for (int i = 0; i < n_small; ++i) {
    const EigDev& e = hp[i];
    const int64_t vecs = small_vec_smem(e.n, e.nvec), all5 = vecs + 4 * (int64_t)e.nvec * (e.n | 1);
    need = std::max(need, all5 <= kVecsSmemCap ? all5 : vecs);
  }
  static thread_local uint64_t attr = 0;  // per host thread and device
  if (tt::first_on_device(attr, ctx->device))
  {
    TT_CUDA(cudaFuncSetAttribute(eigvecs_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kVecsSmemCap)));
    TT_CUDA(cudaFuncSetAttribute(inv_iter_batched, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * 2 * MAX_N)));
  }
  if (n_small > 0) {
    eigvecs_small<<<n_small, small_threads(nsmall_max), sizeof(double) * (size_t)need, ctx->stream>>>(
        dp, G, T, w, Z, work, A, need);
    TT_LAUNCH_CHECK(ctx);
  }
  if (!big.empty()) {
    // the GPU-wide path: inverse iteration, CholeskyQR2, compact-WY
    // back-transformation; problems it flags are redone by the cluster kernel
    if (!iv.empty())
      TT_CUDA(launch(ctx, (int)iv.size(), IV_THREADS, 0, sizeof(double) * 2 * (size_t)nbig_max, n_small > 0, (const void*)inv_iter_batched, db, d_iv, T, w,
                     Z, work));
    for (int pass = 0; pass < 2 && !gm.empty(); ++pass) {
      gram_tiles<<<(unsigned)gm.size(), 256, 0, ctx->stream>>>(db, d_gm, Z, work, flags);
      TT_LAUNCH_CHECK(ctx);
      TT_CUDA(launch_cluster(ctx, cp.cl, CH_THREADS, nbig, 0, (const void*)chol_cluster, db, work, flags, pass == 0 ? 1 : 0));
      trsm_rows<<<(unsigned)ts.size(), TS_THREADS, 0, ctx->stream>>>(db, d_ts, Z, work, flags);
      TT_LAUNCH_CHECK(ctx);
    }
    if (!wy.empty()) {
      wy_factors<<<(unsigned)wy.size(), 256, 0, ctx->stream>>>(db, d_wy, G, T, work, flags);
      TT_LAUNCH_CHECK(ctx);
      wy_apply<<<(unsigned)ap.size(), 512, 0, ctx->stream>>>(db, d_ap, G, Z, work, flags);
      TT_LAUNCH_CHECK(ctx);
    }
    int64_t needc = 0;  // fallback: own eigenvectors in shared memory when they fit, plus 6n of buffers
    for (const EigDev& e : big) {
      const int64_t q = (e.nvec + cp.cl - 1) / cp.cl;
      const int64_t extra = 6 * (int64_t)e.n;
      const int64_t full = q * e.n + extra;
      needc = std::max(needc, full <= cp.vecs_cap ? full : extra);
    }
    TT_CUDA(launch_cluster(ctx, cp.cl, TT, nbig, needc, (const void*)tridiag_eigvecs_cluster, db, G, T, w, Z, work,
                           (int)needc, (const int*)flags));
  }
  tt::pool_free(ctx, buf);
  return TT_OK;
}

}  // extern "C"
