// Device-resident control of tensor_davidsonIT (linalg/tensor_davidson.cpp:193-347).
//
// The host enqueues every iteration of the Davidson loop up front -- products,
// Gram-Schmidt, norms, linear combinations -- and these small control kernels
// carry the decisions that the host loop would otherwise make after reading
// scalars back: the Rayleigh-Ritz step (DIAG of the <= 16 x 16 projected
// matrix, the sign stabilisation, the Ritz coefficients), the convergence
// test, and the bookkeeping of the projected matrix M / Mnext.  Once the loop
// is done (converged, exhausted, or a Gram-Schmidt failure that the host
// handles with its own loop) later control kernels are no-ops, and the host
// reads the state once at the end.  One thread does the work (n <= 16).
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>

#include <cooperative_groups.h>

#include "tt_internal.h"

struct tt_dav_state {
  int done;      // 1 once the loop has ended
  int final_ii;  // iteration at which it ended (-2: Gram-Schmidt failure at fail_ii)
  int fail_ii;
  int iters;
  int refill;      // 1 while the current new vector is a random refill to orthogonalise
  int randomized;  // random refills in this call
  int cur;       // which of buf[0], buf[1] holds M (the other holds Mnext)
  double lambda;
  unsigned long long stamps[TT_DAV_MAX][4];
  double last_lambda, qnorm, gsnorm;
  double buf[2][TT_DAV_MAX * TT_DAV_MAX];
  double evals[TT_DAV_MAX];
  double coef_x[TT_DAV_MAX];      // Ritz vector:   x = sum_k coef_x[k] v[k]
  double coef_q[TT_DAV_MAX + 1];  // residual:      q = sum_k coef_q[k] va[k] + coef_q[ii+1] x
  double H[TT_DAV_MAX][TT_DAV_MAX];  // the projected matrix of the one-launch steps (lower triangle)
};

namespace {

namespace cgx = cooperative_groups;

constexpr int DLD = TT_DAV_MAX + 1;
struct DiagShared {
  double A[TT_DAV_MAX * DLD], V[TT_DAV_MAX * DLD];  // element (i, j) at i + DLD j
  double cs[TT_DAV_MAX / 2], sn[TT_DAV_MAX / 2];
  int pp[TT_DAV_MAX / 2], qq[TT_DAV_MAX / 2];
  int order[TT_DAV_MAX];
};

// DIAG (linalg/lapack_wrapper.cpp:40-54, dsyev semantics) for one warp:
// parallel cyclic Jacobi with the round-robin ordering (every round rotates
// n/2 disjoint index pairs at once; Golub & Van Loan, "Matrix Computations",
// 4th ed., sec. 8.5.5), stopping when the off-diagonal mass falls below
// 1e-32 of the total, as the host DIAG does.  On entry S.A holds the n x n
// matrix; eigenvalues ascending in ev, the eigenvector of ev[j] in column
// S.order[j] of S.V.  All 32 lanes call it.
//
// A chain of latencies: a round is the rotations (two rsqrt in a row in place
// of three divisions and two square roots: cos 2t = |d| / r and sin 2t = h / r
// with d = a_qq - a_pp, h = 2 a_pq, r = |(d, h)|), then one pass that applies
// them to both sides of the 2 x 2 blocks and to V.  An odd n is padded with a
// zero row and column, which no rotation touches.
__device__ void dav_diag_warp(int n, DiagShared& S, double* ev) {
  const int lane = threadIdx.x & 31;
  const int N = n + (n & 1), npair = N / 2;
  // scaled by a power of two, so that no square leaves the range
  double mx = 0.0;
  for (int i = lane; i < n * n; i += 32) mx = fmax(mx, fabs(S.A[i % n + DLD * (i / n)]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const int ex = mx > 0.0 && mx < HUGE_VAL ? ilogb(mx) : 0;
  double fro = 0.0;
  for (int e = lane; e < N * N; e += 32) {
    const int i = e % N, j = e / N;
    const double a = i < n && j < n ? scalbn(S.A[i + DLD * j], -ex) : 0.0;
    S.A[i + DLD * j] = a;
    S.V[i + DLD * j] = i == j ? 1.0 : 0.0;
    fro = fma(a, a, fro);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
  __syncwarp();
  double off = 0.0;
  for (int sweep = 0; sweep < 100; ++sweep) {
    off = 0.0;
    for (int e = lane; e < n * n; e += 32) {
      const int i = e % n, j = e / n;
      const double a = S.A[i + DLD * j];
      if (i != j) off = fma(a, a, off);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
    if (!(off > 1e-32 * fro)) break;  // the same sums on every lane
    for (int r = 0; r < N - 1; ++r) {
      if (lane < npair) {
        // round-robin: player 0 fixed, the others rotate by r
        auto player = [&](int i) {
          int k = i - 1 + r;
          if (k >= N - 1) k -= N - 1;
          return i == 0 ? 0 : k + 1;
        };
        const int a = player(lane), b = player(N - 1 - lane);
        const int p = a < b ? a : b, q = a < b ? b : a;
        const double apq = S.A[p + DLD * q], d = S.A[q + DLD * q] - S.A[p + DLD * p], h = 2.0 * apq;
        const double r2 = fma(d, d, h * h);
        double c = 1.0, sv = 0.0;
        if (apq != 0.0 && r2 > 0.0) {
          const double ri = rsqrt(r2), c2 = fma(0.5 * fabs(d), ri, 0.5), ic = rsqrt(c2);
          c = c2 * ic;
          sv = 0.5 * h * ri * ic;
          if (d < 0.0) sv = -sv;
        }
        S.pp[lane] = p;
        S.qq[lane] = q;
        S.cs[lane] = c;
        S.sn[lane] = sv;
      }
      __syncwarp();
      // A <- J^T A J by the 2 x 2 blocks (pair s, pair t), V <- V J
      for (int it = lane; it < npair * (npair + N); it += 32) {
        const int t = it % npair, u = it / npair;
        const int p = S.pp[t], q = S.qq[t];
        const double c = S.cs[t], sv = S.sn[t];
        if (u < npair) {
          const int ps = S.pp[u], qs = S.qq[u];
          const double cu = S.cs[u], su = S.sn[u];
          double *a0 = S.A + DLD * p, *a1 = S.A + DLD * q;
          const double a = a0[ps], b = a1[ps], e = a0[qs], f = a1[qs];
          const double x0 = c * a - sv * b, x1 = sv * a + c * b, y0 = c * e - sv * f, y1 = sv * e + c * f;
          a0[ps] = cu * x0 - su * y0;
          a1[ps] = u == t && sv != 0.0 ? 0.0 : cu * x1 - su * y1;
          a0[qs] = u == t && sv != 0.0 ? 0.0 : su * x0 + cu * y0;
          a1[qs] = su * x1 + cu * y1;
        } else {
          const int k = u - npair;
          const double vp = S.V[k + DLD * p], vq = S.V[k + DLD * q];
          S.V[k + DLD * p] = c * vp - sv * vq;
          S.V[k + DLD * q] = sv * vp + c * vq;
        }
      }
      __syncwarp();
    }
  }
  if (lane < n) {  // rank by eigenvalue, the first index first on ties
    const double a = S.A[lane + DLD * lane];
    int rank = 0;
    for (int i = 0; i < n; ++i) {
      const double b = S.A[i + DLD * i];
      rank += (b < a || (b == a && i < lane)) ? 1 : 0;
    }
    if (!(off == off)) {  // a NaN in the matrix: everything is
      rank = lane;
      for (int i = 0; i < n; ++i) S.V[i + DLD * lane] = off;
    }
    S.order[rank] = lane;
    ev[rank] = off == off ? scalbn(a, ex) : off;
  }
  __syncwarp();
}

__global__ void dav_begin_kernel(tt_dav_state* st, const double* init_en) {
  if (threadIdx.x != 0) return;
  st->done = 0;
  st->final_ii = -1;
  st->fail_ii = -1;
  st->iters = 0;
  st->cur = 0;
  st->refill = 0;
  st->randomized = 0;
  st->last_lambda = 1000.0;
  const double lam = init_en[0];
  st->lambda = lam;
  st->buf[0][0] = lam;  // M[0] = Mnext[0] = lambda
  st->buf[1][0] = lam;
  st->coef_q[0] = 1.0;  // q = va[0] - lambda v[0]
  st->coef_q[1] = -lam;
}

__global__ void dav_ritz_kernel(tt_dav_state* st, int ii) {
  if (st->done) return;  // uniform: read before anything is written
  const int lane = threadIdx.x & 31;
  const int ni = ii + 1;
  double* M = st->buf[st->cur];
  double* Mn = st->buf[1 - st->cur];
  for (int e = lane; e < ni * ni; e += 32) {
    const int mi = e / ni, mj = e % ni;
    if (mj <= mi) {
      Mn[mj + mi * (ni + 1)] = M[mj + mi * ni];
      Mn[mi + mj * (ni + 1)] = M[mi + mj * ni];
    }
  }
  __shared__ DiagShared S;
  for (int e = lane; e < ni * ni; e += 32) S.A[e % ni + DLD * (e / ni)] = M[e];
  __syncwarp();
  dav_diag_warp(ni, S, st->evals);
  const double* vec = S.V + DLD * S.order[0];
  const double sgn = (vec[0] < 0.0) ? -1.0 : 1.0;  // sign stabilisation (:265-268)
  if (lane <= ii) st->coef_x[lane] = st->coef_q[lane] = sgn * vec[lane];
  if (lane == 0) {
    const double lam = st->evals[0];
    st->lambda = lam;
    st->coef_q[ii + 1] = -lam;
  }
}

__global__ void dav_conv_kernel(tt_dav_state* st, int ii, int maxiter, double tol, const double* qnorm) {
  if (threadIdx.x != 0 || st->done) return;
  const double qn = qnorm[0];
  const double lam = st->lambda;
  const bool converged = (qn < tol && fabs(lam - st->last_lambda) < tol) || qn < fmax(1e-12, tol * 1e-3);
  st->last_lambda = lam;
  st->qnorm = qn;
  st->iters = ii;
  if (qn < 1e-20 || (converged && ii >= 1) || ii == maxiter) {
    st->done = 1;
    st->final_ii = ii;
  }
}

__global__ void dav_row_kernel(tt_dav_state* st, int ii, const double* row, const double* gsnorm) {
  if (threadIdx.x != 0 || st->done) return;
  const double g = gsnorm[0];
  st->gsnorm = g;
  if (!(g >= 1e-10)) {
    // the random refill failed too (the space is exhausted): the loop ends
    // with the current Ritz vector, as the reference does after its retries
    st->done = 1;
    st->final_ii = ii;
    st->fail_ii = ii;
    return;
  }
  const int ni = ii + 1;
  st->cur = 1 - st->cur;  // swap(M, Mnext)
  double* M = st->buf[st->cur];
  const int l = ni;
  for (int k = 0; k < ni + 1; ++k) {
    M[l + k * (ni + 1)] = row[k];
    M[k + l * (ni + 1)] = row[k];
  }
}

// Gram-Schmidt failure inside the loop (linalg/tensor_davidson.cpp:298-316):
// when the projected new vector's norm is below 1e-10 the reference refills it
// with random numbers on the blocks of the previous vector and orthogonalises
// it again; when the vectors already span the problem (ni >= size) the loop
// ends instead.  One launch: every block reads the same norm and decides
// alike (all of them return when there is nothing to do); on a refill each
// thread draws its elements (the counter-based generator of
// tt_vec_fill_random), stores them and accumulates their overlaps with the
// earlier vectors, and the last block (ticket) sums the per-block partials in
// block order into dots and raises st->refill for the conditional
// projection that follows.
constexpr int RF_THREADS = 256;
struct RefillVecs {
  const double* p[TT_DAV_MAX];
};

__device__ __forceinline__ uint64_t rf_mix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void __launch_bounds__(RF_THREADS)
dav_refill_kernel(tt_dav_state* st, int ii, int ni, int maxsize, int64_t n, RefillVecs xs, double* y, int nranges,
                  const int64_t* ranges, uint64_t seed, const double* gsnorm, double* part, double* dots,
                  unsigned int* ticket) {
  if (st->done || gsnorm[0] >= 1e-10) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->refill = 0;
    return;
  }
  if (ni >= maxsize) {  // nothing left to add: the loop ends with the current Ritz vector
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->refill = 0;
      st->done = 1;
      st->final_ii = ii;
      st->fail_ii = ii;
    }
    return;
  }
  double acc[TT_DAV_MAX];
  for (int j = 0; j < ni; ++j) acc[j] = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)RF_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * RF_THREADS) {
    int lo = 0, hi = nranges;  // is i inside one of the sorted [begin, end) ranges?
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (ranges[2 * mid + 1] <= i) lo = mid + 1; else hi = mid;
    }
    double v = 0.0;
    if (lo < nranges && ranges[2 * lo] <= i)
      v = (double)(rf_mix(seed ^ (uint64_t)i * 0xD1B54A32D192ED03ull) >> 11) * 0x1.0p-53;
    y[i] = v;
    for (int j = 0; j < ni; ++j) acc[j] = fma(xs.p[j][i], v, acc[j]);
  }
  __shared__ double red[RF_THREADS / 32][TT_DAV_MAX];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int j = 0; j < ni; ++j) {
    double x = acc[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[w][j] = x;
  }
  __syncthreads();
  if (threadIdx.x < ni) {
    double x = 0.0;
    for (int k = 0; k < RF_THREADS / 32; ++k) x += red[k][threadIdx.x];
    part[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = x;
  }
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < ni) {
    double x = 0.0;
    for (int b = 0; b < (int)gridDim.x; ++b) x += __ldcg(part + (int64_t)threadIdx.x * gridDim.x + b);
    dots[threadIdx.x] = x;
  }
  if (threadIdx.x == 0) {
    st->refill = 1;
    st->randomized++;
    *ticket = 0u;
  }
}

// ---- one Davidson iteration in one launch ------------------------------------
//
// Everything between two products of the Davidson loops: the new row of the
// projected matrix, its diagonalisation, Ritz vector and residual, the test, and
// the next basis vector (linalg/tensor_davidson.cpp:193-347 for block-sparse
// states; DENSE: :74-184, with the diagonal preconditioner and restarts).  One
// cluster of up to 16 CTAs walks the vectors, which are in L2; the sums go through
// the CTAs' shared memory, and every CTA adds them up in the same order and takes
// the same decisions for itself.
//
// At these sizes (a chain's bond) a launch that does almost nothing costs the host
// and the device about 3 us each, and an iteration took eleven of them.  Measured,
// 3 and 6 basis vectors: 16384 elements 20 and 31 us (the calls: 66 and 74), 65536
// 27 and 39 (64 and 75), 262144 46 and 70 (67 and 83), 524288 70 and 111 (79 and 94):
// 16 SMs read more slowly than 148, hence TT_DAV_STEP_MAX.
constexpr int DS_T = 512, DS_W = DS_T / 32, DS_CL = 16;

struct DavStep {
  const double* v[TT_DAV_MAX];   // basis vectors 0..ii
  const double* va[TT_DAV_MAX];  // their products
  const double* y;               // va[ii]
  double* x;                     // Ritz vector
  double* q;                     // residual, then the next basis vector
  const double* D;               // DENSE: the diagonal of the operator
  double* v0;                    // DENSE, last of a restart: v[0] <- x / |x|
  const int64_t* ranges;         // where a random refill may draw
  uint64_t seed;
  int64_t n;
  double tol;
  int ii, maxiter, maxsize, nranges, high, last;
};

template <int N>
struct StepSums {
  double red[DS_W][N], part[2][DS_CL][N], tot[N];
};

// tot[j] = the cluster's sum of acc[j], j < cnt, on every thread after the call
template <int N>
__device__ __forceinline__ void step_sum(double (&acc)[N], int cnt, StepSums<N>& S, int& par, int rank, int CL) {
  cgx::cluster_group cluster = cgx::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (j < cnt) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
      if (lane == 0) S.red[warp][j] = acc[j];
    }
  }
  __syncthreads();
  for (int j = warp; j < cnt; j += DS_W) {
    double s = S.red[lane & (DS_W - 1)][j];
#pragma unroll
    for (int o = DS_W / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < CL) *cluster.map_shared_rank(&S.part[par][rank][j], lane) = s;
  }
  cluster.sync();
  for (int j = warp; j < cnt; j += DS_W) {
    double s = lane < CL ? S.part[par][lane][j] : 0.0;
#pragma unroll
    for (int o = DS_CL / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) S.tot[j] = s;
  }
  __syncthreads();
  par ^= 1;  // the next sums may arrive while these are still read elsewhere
}

template <int NV, bool DENSE>
__global__ void __launch_bounds__(DS_T, 1) dav_step_kernel(tt_dav_state* st, const __grid_constant__ DavStep P) {
  constexpr int N = NV + 3, U = NV <= 4 ? 4 : NV <= 8 ? 2 : 1;  // sums; elements in flight
  __shared__ StepSums<N> S;
  __shared__ DiagShared J;
  __shared__ double ev[TT_DAV_MAX], coef[NV];
  const int ii = P.ii, nv = ii + 1;
  // as after_previous in contract.cu: may start when the blocks of the product before it have ended
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!DENSE && blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    st->stamps[ii][3] = t;
  }
  if (ii > 0 && st->done) return;  // the whole cluster alike: written by an earlier launch
  const double last_lambda = ii > 0 ? st->last_lambda : 1000.0;
  cgx::cluster_group cluster = cgx::this_cluster();
  cluster.sync();  // every CTA has started (and read the state) before one is written to
  const int CL = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x;
  const bool writer = rank == 0 && tid == 0;
  const int64_t n = P.n, e0 = rank * DS_T + tid, step = (int64_t)CL * DS_T;
  int par = 0;
  double acc[N];
  auto clear = [&]() {
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = 0.0;
  };
  // f(e, the basis vectors' element e), U elements in flight
  auto walk = [&](auto pre, auto f) {
    for (int64_t e = e0; e < n; e += U * step) {
      double a[U][NV], b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = e + u * step;
        b[u] = i < n ? pre(i) : 0.0;
#pragma unroll
        for (int j = 0; j < NV; ++j) a[u][j] = j < nv && i < n ? P.v[j][i] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (e + u * step < n) f(e + u * step, a[u], b[u]);
    }
  };
  auto overlaps = [&](double b, const double (&a)[NV]) {
#pragma unroll
    for (int j = 0; j < NV; ++j) acc[j] = fma(a[j], b, acc[j]);
  };
  // ---- the new row of the projected matrix ----
  clear();
  walk([&](int64_t i) { return P.y[i]; }, [&](int64_t, const double (&a)[NV], double b) { overlaps(b, a); });
  step_sum(acc, nv, S, par, rank, CL);
  // ---- its lowest (highest) eigenpair ----
  if (tid < 32) {
    for (int e = tid; e < nv * nv; e += 32) {
      const int i = e % nv, j = e / nv, hi = i > j ? i : j, lo = i > j ? j : i;
      J.A[i + DLD * j] = hi == ii ? S.tot[lo] : st->H[hi][lo];
    }
    __syncwarp();
    dav_diag_warp(nv, J, ev);
    const int which = DENSE && P.high ? ii : 0;
    const double* vec = J.V + DLD * J.order[which];
    const double sgn = !DENSE && vec[0] < 0.0 ? -1.0 : 1.0;  // sign stabilisation (:265-268)
    if (tid < nv) {
      coef[tid] = sgn * vec[tid];
      if (rank == 0) st->H[ii][tid] = S.tot[tid];
    }
  }
  __syncthreads();
  const double lambda = ev[DENSE && P.high ? ii : 0];
  // ---- Ritz vector, residual, its norm and its overlaps with the basis ----
  clear();
  for (int64_t e = e0; e < n; e += U * step) {
    double a[U][NV], b[U][NV], d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = e + u * step;
      d[u] = DENSE && i < n ? P.D[i] : 0.0;
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        a[u][j] = j < nv && i < n ? P.v[j][i] : 0.0;
        b[u][j] = j < nv && i < n ? P.va[j][i] : 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = e + u * step;
      if (i >= n) continue;
      double xs = 0.0, qs = 0.0;
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const double c = j < nv ? coef[j] : 0.0;
        xs = fma(c, a[u][j], xs);
        qs = fma(c, b[u][j], qs);
      }
      qs = fma(-lambda, xs, qs);
      acc[NV] = fma(qs, qs, acc[NV]);
      if (DENSE) {
        if (d[u] != lambda) qs /= d[u] - lambda;  // elemWiseDivide (:25-36)
        acc[NV + 1] = fma(qs, qs, acc[NV + 1]);
        acc[NV + 2] = fma(xs, xs, acc[NV + 2]);
      }
      overlaps(qs, a[u]);
      if (DENSE ? P.last : ii > 0) P.x[i] = xs;
      if (!DENSE || !P.last) P.q[i] = qs;
    }
  }
  step_sum(acc, N, S, par, rank, CL);
  const double qnorm = sqrt(S.tot[NV]);
  double inv = 1.0;
  // DENSE: there is no further direction.  The restart ends with the present Ritz
  // vector in x and, normalised, in v[0]; its later steps do nothing.
  auto end_restart = [&]() {
    const double scale = 1.0 / sqrt(S.tot[NV + 2]);
    walk([&](int64_t) { return 0.0; },
         [&](int64_t i, const double (&a)[NV], double) {
           double xs = 0.0;
#pragma unroll
           for (int j = 0; j < NV; ++j) xs = fma(j < nv ? coef[j] : 0.0, a[j], xs);
           P.x[i] = xs;
           P.v0[i] = xs * scale;
         });
    if (writer) st->done = 1;
  };
  if (DENSE) {
    if (writer) {
      st->last_lambda = lambda;
      st->qnorm = qnorm;
      st->done = 0;
    }
    if (P.last) {
      inv = 1.0 / sqrt(S.tot[NV + 2]);
      for (int64_t i = e0; i < n; i += step) P.v0[i] = P.x[i] * inv;
      return;
    }
    if (S.tot[NV + 1] == 0.0) return end_restart();  // the Ritz vector is an eigenvector
    inv = 1.0 / sqrt(S.tot[NV + 1]);
  } else {
    const bool converged =
        (qnorm < P.tol && fabs(lambda - last_lambda) < P.tol) || qnorm < fmax(1e-12, P.tol * 1e-3);
    const bool ends = qnorm < 1e-20 || (converged && ii >= 1) || ii == P.maxiter;
    if (writer) {
      st->lambda = lambda;
      st->last_lambda = lambda;
      st->qnorm = qnorm;
      st->iters = ii;
      st->done = ends;
      st->final_ii = ends ? ii : -1;
      if (ii == 0) {
        st->fail_ii = -1;
        st->randomized = 0;
      }
    }
    if (ends) return;
  }
  // ---- Gram-Schmidt: q <- scale q - sum_j (scale o_j) v_j and its norm ----
  auto project = [&](double scale) {
    double o[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) o[j] = j < nv ? scale * S.tot[j] : 0.0;
    double norm2 = 0.0;
    walk([&](int64_t i) { return P.q[i]; },
         [&](int64_t i, const double (&a)[NV], double b) {
           b *= scale;
#pragma unroll
           for (int j = 0; j < NV; ++j) b = fma(-o[j], a[j], b);
           P.q[i] = b;
           norm2 = fma(b, b, norm2);
         });
    clear();
    acc[0] = norm2;
    step_sum(acc, 1, S, par, rank, CL);
    return sqrt(S.tot[0]);
  };
  double g = project(inv);
  if (DENSE) {
    // q was a unit vector: a small remainder is mostly the cancellation's rounding
    // and is projected again.  Rounding that lies outside the basis is as good a
    // direction as a random one and keeps its length; of rounding that lies in it, a
    // basis that spans the space, nothing is left time after time.
    for (int again = 0; g < 0.1; ++again) {
      if (again == 2 || g == 0.0) return end_restart();
      clear();
      walk([&](int64_t i) { return P.q[i]; }, [&](int64_t, const double (&a)[NV], double b) { overlaps(b, a); });
      step_sum(acc, nv, S, par, rank, CL);
      g = project(1.0 / g);
    }
  } else if (!(g >= 1e-10)) {
    // Gram-Schmidt failure (:298-316): random numbers on the blocks of the vector
    // before, projected once more; the loop ends when the vectors already span the
    // problem or that fails too
    if (nv < P.maxsize) {
      clear();
      walk([&](int64_t) { return 0.0; },
           [&](int64_t i, const double (&a)[NV], double) {
             int lo = 0, hi = P.nranges;  // is i inside one of the sorted [begin, end) ranges?
             while (lo < hi) {
               const int mid = (lo + hi) >> 1;
               if (P.ranges[2 * mid + 1] <= i) lo = mid + 1; else hi = mid;
             }
             double v = 0.0;
             if (lo < P.nranges && P.ranges[2 * lo] <= i)
               v = (double)(rf_mix(P.seed ^ (uint64_t)i * 0xD1B54A32D192ED03ull) >> 11) * 0x1.0p-53;
             P.q[i] = v;
             overlaps(v, a);
           });
      step_sum(acc, nv, S, par, rank, CL);
      g = project(1.0);
      if (writer) st->randomized++;
    }
    if (!(g >= 1e-10)) {
      if (writer) {
        st->done = 1;
        st->final_ii = ii;
        st->fail_ii = ii;
      }
      return;
    }
  }
  if (!DENSE && writer) st->gsnorm = g;
  inv = 1.0 / g;
  for (int64_t i = e0; i < n; i += step) P.q[i] *= inv;
}

}  // namespace

extern "C" {

int tt_dav_state_create(tt_ctx* ctx, tt_dav_state** out) {
  TT_REQUIRE(ctx && out, "tt_dav_state_create: null argument");
  tt_dav_state* s = nullptr;
  TT_CUDA(cudaMalloc(&s, sizeof(tt_dav_state)));
  TT_CUDA(cudaMemsetAsync(s, 0, sizeof(tt_dav_state), ctx->stream));
  *out = s;
  return TT_OK;
}

int tt_dav_state_destroy(tt_ctx* ctx, tt_dav_state* st) {
  (void)ctx;
  if (st) cudaFree(st);
  return TT_OK;
}

int tt_dav_coefficients(tt_dav_state* st, double** coef_x, double** coef_q) {
  TT_REQUIRE(st && coef_x && coef_q, "tt_dav_coefficients: null argument");
  *coef_x = st->coef_x;
  *coef_q = st->coef_q;
  return TT_OK;
}

int tt_dav_begin(tt_ctx* ctx, tt_dav_state* st, const double* d_init_energy) {
  TT_REQUIRE(ctx && st && d_init_energy, "tt_dav_begin: null argument");
  dav_begin_kernel<<<1, 32, 0, ctx->stream>>>(st, d_init_energy);
  TT_LAUNCH_CHECK(ctx);
  return TT_OK;
}

int tt_dav_ritz(tt_ctx* ctx, tt_dav_state* st, int ii) {
  TT_REQUIRE(ctx && st && ii >= 1 && ii + 1 < TT_DAV_MAX, "tt_dav_ritz: bad argument");
  dav_ritz_kernel<<<1, 32, 0, ctx->stream>>>(st, ii);
  TT_LAUNCH_CHECK(ctx);
  return TT_OK;
}

int tt_dav_converged(tt_ctx* ctx, tt_dav_state* st, int ii, int maxiter, double tol, const double* d_qnorm) {
  TT_REQUIRE(ctx && st && d_qnorm && ii >= 0 && maxiter + 1 < TT_DAV_MAX, "tt_dav_converged: bad argument");
  dav_conv_kernel<<<1, 32, 0, ctx->stream>>>(st, ii, maxiter, tol, d_qnorm);
  TT_LAUNCH_CHECK(ctx);
  return TT_OK;
}

int tt_dav_add_row(tt_ctx* ctx, tt_dav_state* st, int ii, const double* d_row, const double* d_gsnorm) {
  TT_REQUIRE(ctx && st && d_row && d_gsnorm && ii >= 0 && ii + 2 < TT_DAV_MAX, "tt_dav_add_row: bad argument");
  dav_row_kernel<<<1, 32, 0, ctx->stream>>>(st, ii, d_row, d_gsnorm);
  TT_LAUNCH_CHECK(ctx);
  return TT_OK;
}

int tt_dav_gs_refill(tt_ctx* ctx, tt_dav_state* st, int ii, int ni, int maxsize, int64_t n,
                     const double* const* xs, double* y, int nranges, const int64_t* d_ranges, uint64_t seed,
                     const double* d_gsnorm, double* d_dots) {
  TT_REQUIRE(ctx && st && xs && y && d_gsnorm && d_dots && (nranges == 0 || d_ranges),
             "tt_dav_gs_refill: null argument");
  TT_REQUIRE(ni >= 1 && ni <= TT_DAV_MAX && ii >= 0 && n >= 0, "tt_dav_gs_refill: bad argument");
  RefillVecs v;
  for (int j = 0; j < ni; ++j) v.p[j] = xs[j];
  const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((n + RF_THREADS - 1) / RF_THREADS,
                                                                  4 * (int64_t)ctx->num_sms));
  double* part = tt::partials(ctx, nb * ni);
  if (!part) return tt::fail(TT_ERR_OOM, "tt_dav_gs_refill: reduction scratch");
  dav_refill_kernel<<<nb, RF_THREADS, 0, ctx->stream>>>(st, ii, ni, maxsize, n, v, y, nranges, d_ranges, seed,
                                                        d_gsnorm, part, d_dots, ctx->d_ticket);
  TT_LAUNCH_CHECK(ctx);
  return TT_OK;
}

extern "C++" {
template <bool DENSE>
static int launch_step(tt_ctx* ctx, tt_dav_state* st, const DavStep& P) {
  const int nv = P.ii + 1;
  const void* kernel = nv <= 4   ? (const void*)dav_step_kernel<4, DENSE>
                       : nv <= 8 ? (const void*)dav_step_kernel<8, DENSE>
                                 : (const void*)dav_step_kernel<TT_DAV_MAX, DENSE>;
  // two elements a thread before the cluster grows (3000 elements, 3 and 6 vectors: 16.7
  // and 27.0 us; one element 16.5 and 26.5, four 17.2 and 29.3)
  int cl = 1;
  while (cl < DS_CL && (int64_t)cl * DS_T * 2 < P.n) cl *= 2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)cl);
  cfg.blockDim = dim3(DS_T);
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  if (cl > 8) {
    // per host thread and device: whether clusters of 16 fit (8 always may)
    static thread_local uint64_t asked[3] = {0, 0, 0}, fits[3] = {0, 0, 0};
    const int which = nv <= 4 ? 0 : nv <= 8 ? 1 : 2;
    const uint64_t bit = (uint64_t)1 << (ctx->device & 63);
    if (tt::first_on_device(asked[which], ctx->device)) {
      int nc = 0;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
          cudaOccupancyMaxActiveClusters(&nc, kernel, &cfg) == cudaSuccess && nc >= 1)
        fits[which] |= bit;
      else
        cudaGetLastError();
    }
    if (!(fits[which] & bit)) {
      cl = 8;
      at[0].val.clusterDim.x = cl;
      cfg.gridDim = dim3((unsigned)cl);
    }
  }
  void* argv[] = {(void*)&st, (void*)&P};
  TT_CUDA(cudaLaunchKernelExC(&cfg, kernel, argv));
  TT_LAUNCH_CHECK(ctx);
  return TT_OK;
}
}  // extern "C++"

int tt_dav_step(tt_ctx* ctx, tt_dav_state* st, int ii, int maxiter, double tol, int maxsize, int64_t n,
                const double* const* vs, const double* const* vas, double* x, double* q, int nranges,
                const int64_t* d_ranges, uint64_t seed) {
  TT_REQUIRE(ctx && st && vs && vas && x && q && (nranges == 0 || d_ranges), "tt_dav_step: null argument");
  TT_REQUIRE(ii >= 0 && ii <= maxiter && maxiter + 2 <= TT_DAV_MAX && n >= 1, "tt_dav_step: bad argument");
  DavStep P = {};
  for (int j = 0; j <= ii; ++j) {
    P.v[j] = vs[j];
    P.va[j] = vas[j];
  }
  P.y = vas[ii];
  P.x = x;
  P.q = q;
  P.ranges = d_ranges;
  P.nranges = nranges;
  P.seed = seed;
  P.n = n;
  P.tol = tol;
  P.ii = ii;
  P.maxiter = maxiter;
  P.maxsize = maxsize;
  return launch_step<false>(ctx, st, P);
}

int tt_dav_step_dense(tt_ctx* ctx, tt_dav_state* st, int j, int m, int high, int64_t n, double* const* vs,
                      const double* const* vas, const double* D, double* x) {
  TT_REQUIRE(ctx && st && vs && vas && D && x, "tt_dav_step_dense: null argument");
  TT_REQUIRE(j >= 0 && j < m && m <= TT_DAV_MAX && n >= 1, "tt_dav_step_dense: bad argument");
  DavStep P = {};
  for (int k = 0; k <= j; ++k) {
    P.v[k] = vs[k];
    P.va[k] = vas[k];
  }
  P.y = vas[j];
  P.x = x;
  P.last = j == m - 1;
  P.q = P.last ? nullptr : vs[j + 1];
  P.v0 = vs[0];
  P.D = D;
  P.n = n;
  P.ii = j;
  P.high = high;
  return launch_step<true>(ctx, st, P);
}

int tt_dav_read_dense(tt_ctx* ctx, const tt_dav_state* st, double* eval, double* r_norm) {
  TT_REQUIRE(ctx && st && eval && r_norm, "tt_dav_read_dense: null argument");
  double h[2];
  static_assert(offsetof(tt_dav_state, qnorm) == offsetof(tt_dav_state, last_lambda) + sizeof(double), "read at once");
  int rc = tt_memcpy_d2h(ctx, h, &st->last_lambda, sizeof(h));
  if (rc != TT_OK) return rc;
  *eval = h[0];
  *r_norm = h[1];
  return TT_OK;
}

int tt_dav_refill_flag(tt_dav_state* st, const int** d_flag) {
  TT_REQUIRE(st && d_flag, "tt_dav_refill_flag: null argument");
  *d_flag = &st->refill;
  return TT_OK;
}

int tt_dav_stamp_slots(tt_dav_state* st, int i, uint64_t** d_slots) {
  TT_REQUIRE(st && d_slots && i >= 0 && i < TT_DAV_MAX, "tt_dav_stamp_slots: bad argument");
  *d_slots = reinterpret_cast<uint64_t*>(st->stamps[i]);
  return TT_OK;
}

int tt_dav_read(tt_ctx* ctx, const tt_dav_state* st, tt_dav_result* out) {
  return tt_dav_read_stamped(ctx, st, out, nullptr);
}

int tt_dav_read_stamped(tt_ctx* ctx, const tt_dav_state* st, tt_dav_result* out, uint64_t* stamps) {
  TT_REQUIRE(ctx && st && out, "tt_dav_read: null argument");
  // one synchronising read of the header: the flags, the Ritz value, the clocks
  constexpr size_t kHead = offsetof(tt_dav_state, stamps), kAll = kHead + sizeof(tt_dav_state::stamps);
  alignas(8) unsigned char h[kAll];
  int rc = tt_memcpy_d2h(ctx, h, st, stamps ? kAll : kHead);
  if (rc != TT_OK) return rc;
  if (stamps) std::memcpy(stamps, h + kHead, kAll - kHead);
  tt_dav_state head;
  std::memcpy(&head, h, kHead);
  out->done = head.done;
  out->final_ii = head.final_ii;
  out->fail_ii = head.fail_ii;
  out->iters = head.iters;
  out->randomized = head.randomized;
  out->lambda = head.lambda;
  return TT_OK;
}

}  // extern "C"
