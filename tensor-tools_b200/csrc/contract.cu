// Grouped block-sparse contraction: every (output block, block pair) GEMM of
// one qtensor::operator* (qtensor/qtensor.cpp:652-726) in a single launch.
//
// FP64 path: 64x64 CTA tiles, BK=16, 3-stage cp.async pipeline, four warps
// of 32x32 built from mma.sync m16n8k8 f64 (DMMA), a tile's k range shared by
// a cluster of CTAs where the plan has few tiles.  Operands are gathered
// through the strides of the tensor blocks (or per-pair offset tables, where
// the modes of a row or column do not merge into one stride), so any index
// permutation of the contraction is handled without a transpose pass; the
// tables are expanded on the device from the pair descriptors when the plan is
// built.
#include <cooperative_groups.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cstring>
#include <functional>
#include <map>
#include <numeric>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "tt_internal.h"

namespace {

constexpr int BM = 64;
constexpr int BN = 64;
constexpr int BK = 16;
constexpr int STAGES = 3;
constexpr int MT = BM / 32;  // 16-row parts of a warp's tile (2 x THREADS / 64 warps)
constexpr int THREADS = 128;
constexpr int WN = BN / (THREADS / 64);  // columns of a warp's tile
constexpr int NT = WN / 8;               // its 8-column parts
constexpr int STAGE_EL = (BM + BN) * BK;  // elements of a stage: A's rows, then B's
constexpr size_t SMEM_BYTES = sizeof(double) * STAGES * STAGE_EL;
constexpr int PAIR_BATCH = 16;   // pair descriptors staged in shared memory at a time
constexpr int SPLIT_MAX = 8;     // most CTAs (one portable cluster) sharing a tile's k range

struct PairDev {
  int64_t a_off, b_off;
  int32_t m, n, k;
  int32_t rowA, colA, rowB, colB;  // offsets of the tables in the table buffer
  int32_t a_mfast, b_kfast;        // unit stride along m (A) / along k (B)
  // the stride of A's rows and columns and of B's rows and columns where all
  // modes merge into one (offset = index * stride); NO_STRIDE: use the table
  int32_t a_rs, a_ks, b_ks, b_cs;
};
constexpr int32_t NO_STRIDE = INT_MIN;

struct TaskDev {
  int32_t out;
  int32_t m0, n0;
  int32_t p_begin, p_end;
};

struct DTask {  // one output tile of grouped_dgemm, with its output block
  int64_t c_off;
  int32_t m, n, ldc;
  int32_t m0, n0, p_begin, p_end;
  int32_t chunks;  // BK-wide k chunks over its pairs
};

struct OutDev {
  int64_t c_off;
  int32_t m, n, ldc;
};

struct TableJob {  // one of the four offset tables of a pair
  int32_t dst;     // offset in the table buffer
  int32_t len;
  int32_t nmodes;
  int32_t dims[TT_MAX_MODES];
  int64_t strides[TT_MAX_MODES];
};

__global__ void expand_tables(const TableJob* jobs, int njobs, int32_t* tab) {
  int j = blockIdx.x;
  if (j >= njobs) return;
  const TableJob& J = jobs[j];
  for (int i = threadIdx.x; i < J.len; i += blockDim.x) {
    int64_t off = 0;
    int r = i;
    for (int d = 0; d < J.nmodes; ++d) {
      int q = r / J.dims[d];
      off += (int64_t)(r - q * J.dims[d]) * J.strides[d];
      r = q;
    }
    tab[J.dst + i] = (int32_t)off;
  }
}

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem, bool pred) {
  unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
  int src_bytes = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(gmem),
               "r"(src_bytes));
}
__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
  unsigned saddr = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(saddr), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// D += A B, m16n8k8 FP64 (DMMA).  Lane 4g + t holds
// A[g][t], A[g+8][t], A[g][t+4], A[g+8][t+4]; B[t][g], B[t+4][g];
// D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1].
__device__ __forceinline__ void dmma_k8(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
// Element (r, k) of an operand's stage: rows of 64 along m or n (KF false), or
// rows of 16 along k (KF true), whichever the operand is contiguous in, so a
// warp's 8-byte copies write consecutive shared memory.  A fragment's lane t
// takes k = 2t and 2t + 1 (any assignment does, the same for A and B), in KF
// form with one 16-byte load.  The XOR spreads a fragment load over the banks
// without padding: a half-warp's 4 rows x 4 k (8-byte loads), a quarter-warp's
// 2 rows x 4 pairs of k (16-byte loads) touch every bank once.
template <bool KF, int R>
__device__ __forceinline__ int stage_at(int r, int k) {
  return KF ? r * BK + (k ^ ((r & 1) << 3)) : k * R + (r ^ ((k & 6) << 1));
}

// rows r and k = kk + 2t, kk + 2t + 1 of a stage
template <bool KF, int R>
__device__ __forceinline__ void frag2(const double* st, int r, int kk, int t4, double& lo, double& hi) {
  if (KF) {
    const double2 v = *reinterpret_cast<const double2*>(st + stage_at<true, R>(r, kk + 2 * t4));
    lo = v.x;
    hi = v.y;
  } else {
    lo = st[stage_at<false, R>(r, kk + 2 * t4)];
    hi = st[stage_at<false, R>(r, kk + 2 * t4 + 1)];
  }
}

// one k chunk of a warp's 32x32 tile, k8 (1 or 2) steps of 8; mt / nt: its
// 16-row and 8-column parts that hold output (FULL: all of them)
template <bool AKF, bool BKF, bool FULL>
__device__ __forceinline__ void dgemm_chunk(const double* as, const double* bs, double (&acc)[MT][NT][4], int k8,
                                            int wm, int wn, int g, int t4, int mt, int nt) {
#pragma unroll
  for (int kk = 0; kk < BK; kk += 8) {
    if (kk >= 8 * k8) break;
    double a[MT][4], b[NT][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) frag2<AKF, BM>(as, wm + i * 16 + h * 8 + g, kk, t4, a[i][h], a[i][h + 2]);
#pragma unroll
    for (int j = 0; j < NT; ++j) frag2<BKF, BN>(bs, wn + j * 8 + g, kk, t4, b[j][0], b[j][1]);
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
        if (FULL || (i < mt && j < nt)) dmma_k8(acc[i][j], a[i], b[j]);
  }
}

// One operand's chunk (R rows x BK k) into its stage: 8-byte copies,
// along the operand's contiguous direction, the thread's other index
// fixed; rows past the block and k past the pair are zero-filled.  rs / ks:
// strides, or NO_STRIDE for the table.  The copies of a chunk inside the block
// need one address addition each.
template <bool KF, int R>
__device__ __forceinline__ void load_chunk(double* st, const double* __restrict__ X, const int32_t* __restrict__ tab,
                                           int row_tab, int k_tab, int32_t rs, int32_t ks, int r0, int rows, int k0,
                                           int K, int tid) {
  constexpr int DV = KF ? THREADS / BK : THREADS / R;         // step of the walked index
  constexpr int NQ = KF ? R / DV : BK / DV;                   // copies per thread
  const int fi = KF ? k0 + (tid & 15) : r0 + (tid & (R - 1));      // fixed index (k, or row)
  const int vi = KF ? r0 + (tid >> 4) : k0 + tid / R;      // first walked index (row, or k)
  const int fn = KF ? K : rows, vn = KF ? rows : K;           // their ends
  const int32_t fs = KF ? ks : rs, vs = KF ? rs : ks;
  const bool fv = fi < fn;
  const double* base = X + (fs != NO_STRIDE ? (int64_t)fi * fs : (int64_t)(fv ? tab[(KF ? k_tab : row_tab) + fi] : 0));
  auto dst = [&](int q) {
    return st + (KF ? stage_at<true, R>((tid >> 4) + DV * q, tid & 15) : stage_at<false, R>(tid & (R - 1), tid / R + DV * q));
  };
  if (vs != NO_STRIDE) {
    const double* p = base + (int64_t)vi * vs;
    const int64_t step = (int64_t)DV * vs;
    if (r0 + R <= rows && k0 + BK <= K) {  // the whole CTA alike
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        cp_async8(dst(q), p);
        p += step;
      }
    } else {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const bool ok = fv && vi + DV * q < vn;
        cp_async8(dst(q), ok ? p : X, ok);
        p += step;
      }
    }
  } else {
    const int32_t* vt = tab + (KF ? row_tab : k_tab) + vi;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const bool ok = fv && vi + DV * q < vn;
      cp_async8(dst(q), ok ? base + vt[DV * q] : X, ok);
    }
  }
}

// A contraction is one of a chain of small launches.  It is launched so that it may
// start when the blocks of the kernel before it have ended; it waits here for that
// kernel's memory before it touches anything but its own plan, which an earlier copy
// wrote.  (A kernel that let the next one in from its own start lost 5 % at
// m = 1400.)  The pointers to what plain loads read pass through the wait: no read
// through a __restrict__ argument is moved above it (asynchronous copies are not
// moved; rows_dgemm's loads of A have a line of their own).  The stamp is the device's clock at that point.  Nine
// launches of three products at a chain's m = 128: 86 -> 68 us.
__device__ __forceinline__ void after_previous(const int32_t* __restrict__& tab, unsigned long long* stamp) {
  asm volatile("griddepcontrol.wait;" : "+l"(tab) : : "memory");
  if (stamp && blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    *stamp = t;
  }
}

// A cluster of CTAs (one, where the plan has tiles enough to fill the GPU)
// takes one output tile; its CTAs share the tile's k chunks evenly, in order,
// and add their partial tiles through distributed shared memory, CTA 0's
// first, so the result does not depend on timing.  The chunks of all pairs of
// a tile form one stream through the ring: the copies of a pair's first chunks
// are in flight while the previous pair's last ones are multiplied.
//
// Bound by the FP64 tensor pipe (37 TFLOP/s when it is fed from registers); the
// copies' issue slots and shared-memory wavefronts hide behind it only in part:
// on the environment update's products (25 GFLOP, blocks of 3 to 545) the pipe is
// active 75 % of the time, 83 % with the copies left out.  64 x 64 tiles of four
// warps with four CTAs per SM measured best: 128 x 64 tiles, eight warps per tile
// or a fourth stage were 3 to 14 % slower.  Measured against offset tables read
// for every element, padded stages and m8n8k4 fragments: env update at bond
// dimension 2048 1154 -> 975 us per product; R product at 1400 1110 -> 730 us,
// where the tile's k range is now shared.
__global__ void __launch_bounds__(THREADS, 4)
grouped_dgemm(const DTask* __restrict__ tasks,
              const PairDev* __restrict__ pairs, const int32_t* __restrict__ tab,
              const double* __restrict__ A, const double* __restrict__ B,
              double* __restrict__ C, double alpha, int split, unsigned long long* stamp) {
  extern __shared__ double smem[];  // [STAGES][A stage, B stage]
  __shared__ PairDev sp[PAIR_BATCH];
  __shared__ int32_t s_meta[STAGES];  // of the chunk in a stage: its 8-wide k steps, and its operands' directions

  // after_previous, written out (the call: 2920 us instead of 2865 for two products at m = 1400)
  asm volatile("griddepcontrol.wait;" : "+l"(tab) : : "memory");
  if (stamp && blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    *stamp = t;
  }
  const DTask task = tasks[blockIdx.x / split];
  const int rank = blockIdx.x % split;  // its place in the cluster (clusters are consecutive blocks)
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int wm = (warp & 1) * (BM / 2);
  const int wn = (warp >> 1) * WN;
  const int g = lane >> 2;  // groupID
  const int t4 = lane & 3;  // thread in group
  // parts of this warp's tile that hold output
  const int mt = max(0, min(MT, (task.m - task.m0 - wm + 15) >> 4));
  const int nt = mt == 0 ? 0 : max(0, min(NT, (task.n - task.n0 - wn + 7) >> 3));
  const bool full = mt == MT && nt == NT;

  double acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

  // the loader's place in the stream: pair lp (its descriptor in sp), its chunk lc of lnch
  int lp = task.p_begin, base = task.p_begin, lc = 0, lnch = 0;
  auto stage_pairs = [&](int from) {  // every thread alike
    __syncthreads();
    constexpr int W = sizeof(PairDev) / 4;
    const int cnt = min(PAIR_BATCH, task.p_end - from) * W;
    for (int i = tid; i < cnt; i += THREADS)
      reinterpret_cast<int32_t*>(sp)[i] = reinterpret_cast<const int32_t*>(pairs + from)[i];
    __syncthreads();
    base = from;
  };
  const int c0 = (int)((int64_t)task.chunks * rank / split), c1 = (int)((int64_t)task.chunks * (rank + 1) / split);
  const int nch = c1 - c0;
  if (nch > 0) {
    stage_pairs(lp);
    lc = c0;
    while (true) {  // the pair that holds chunk c0
      lnch = (sp[lp - base].k + BK - 1) / BK;
      if (lc < lnch) break;
      lc -= lnch;
      if (++lp - base == PAIR_BATCH) stage_pairs(lp);
    }
  }
  auto load_next = [&](int stage) {
    while (lc == lnch) {  // on to the next pair
      if (++lp - base == PAIR_BATCH) stage_pairs(lp);
      lnch = (sp[lp - base].k + BK - 1) / BK;
      lc = 0;
    }
    const PairDev& P = sp[lp - base];
    const int k0 = lc * BK, K = P.k;
    const bool akf = !P.a_mfast, bkf = P.b_kfast;
    double* as = smem + stage * STAGE_EL;
    double* bs = as + BM * BK;
    if (akf) load_chunk<true, BM>(as, A + P.a_off, tab, P.rowA, P.colA, P.a_rs, P.a_ks, task.m0, P.m, k0, K, tid);
    else load_chunk<false, BM>(as, A + P.a_off, tab, P.rowA, P.colA, P.a_rs, P.a_ks, task.m0, P.m, k0, K, tid);
    if (bkf) load_chunk<true, BN>(bs, B + P.b_off, tab, P.colB, P.rowB, P.b_cs, P.b_ks, task.n0, P.n, k0, K, tid);
    else load_chunk<false, BN>(bs, B + P.b_off, tab, P.colB, P.rowB, P.b_cs, P.b_ks, task.n0, P.n, k0, K, tid);
    if (tid == 0) s_meta[stage] = (K - k0 > 8 ? 2 : 1) | (akf ? 4 : 0) | (bkf ? 8 : 0);
    ++lc;
  };

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nch) load_next(s);
    cp_async_commit();
  }
  for (int c = 0; c < nch; ++c) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    const int stage = c % STAGES;
    const int meta = s_meta[stage];
    const int k8 = meta & 3;
    const double* as = smem + stage * STAGE_EL;
    const double* bs = as + BM * BK;
    if (full) {
      switch (meta >> 2) {
        case 0: dgemm_chunk<false, false, true>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
        case 1: dgemm_chunk<true, false, true>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
        case 2: dgemm_chunk<false, true, true>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
        default: dgemm_chunk<true, true, true>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
      }
    } else if (nt > 0) {
      switch (meta >> 2) {
        case 0: dgemm_chunk<false, false, false>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
        case 1: dgemm_chunk<true, false, false>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
        case 2: dgemm_chunk<false, true, false>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
        default: dgemm_chunk<true, true, false>(as, bs, acc, k8, wm, wn, g, t4, mt, nt); break;
      }
    }
    if (c + STAGES - 1 < nch) load_next((c + STAGES - 1) % STAGES);
    cp_async_commit();
  }
  cp_async_wait<0>();

  // epilogue: C tile = alpha * acc (blocks without pairs get zeros)
  double* Cb = C + task.c_off;
  if (split == 1) {
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int m = task.m0 + wm + i * 16 + (e >> 1) * 8 + g;
          const int n = task.n0 + wn + j * 8 + 2 * t4 + (e & 1);
          if (m < task.m && n < task.n) Cb[m + (int64_t)task.ldc * n] = alpha * acc[i][j][e];
        }
    return;
  }
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __syncthreads();  // the ring is free: this CTA's partial tile goes there, column-major
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        smem[(wm + i * 16 + (e >> 1) * 8 + g) + BM * (wn + j * 8 + 2 * t4 + (e & 1))] = acc[i][j][e];
  cluster.sync();
  const int per = BN / split;  // columns this CTA adds up
  for (int el = tid; el < BM * per; el += THREADS) {
    const int at = BM * per * rank + el;
    double s = 0.0;
    for (int q = 0; q < split; ++q) s += *cluster.map_shared_rank(smem + at, q);
    const int m = task.m0 + at % BM, n = task.n0 + at / BM;
    if (m < task.m && n < task.n) Cb[m + (int64_t)task.ldc * n] = alpha * s;
  }
  cluster.sync();  // no CTA leaves while another reads its partial tile
}

// ---------------------------------------------------------------------------
// Narrow FP64 path: contractions whose output blocks have at most NR_N columns
// and whose pairs contract at most NR_K elements -- the middle contraction of
// H_eff*x and of the environment update, (a' b) x (w s1 s2) times (w s1 s2) x
// (s1' s2' w'), with rows a' b in the hundreds of thousands and k, n the MPO
// link sector widths.  It is bound by reading T1 and writing T2.
//
// Output blocks that contract the same A blocks (the (s1' s2' w') sectors fed
// by one set of T1 blocks) form chunks of at most NR_N columns; the A blocks of
// a chunk, one after another, are its k.  A warp takes 32 rows of a chunk at a
// time: lane r copies row r of every k to shared memory (8-byte cp.async: 256
// contiguous bytes per k for a unit row stride), one tile ahead of the one that
// the m8n8k4 FP64 tensor-core products multiply with the chunk's B (staged once
// per CTA) into all the chunk's columns.  So T1 is read once per NR_N columns that
// contract the same A blocks (an output block that shares only some of them is in a
// chunk of its own and reads them again), no column or k is padded by more than a
// fragment, and after the staging a warp needs no barrier.
// Measured on the middle contraction (read T1, write T2): bond dimension 3072
// (2.03 GB) 1131 -> 620 us (1.8 -> 3.3 TB/s), 1400 (0.42 GB) 246 -> 119 us,
// against a thread per row with the products as FP64 FMAs, 16 columns a time.
// What is left is instruction issue (at 1400: IPC 1.8, the tensor pipe active for
// 41 % of the launch, DRAM at 40 % of its peak).
// Buffers of 16 k with four CTAs per SM measured best: 32 k (three CTAs) 662 us,
// five CTAs at 96 registers 740 us; A loaded straight into the fragments 853 us.
constexpr int NR_N = 32;          // columns of a chunk, at most
constexpr int NR_K = 64;          // k of a pair, at most
constexpr int NR_KTOT = 256;      // k of a chunk, at most (its B is staged whole; 106 KB with 32 columns, two CTAs)
// row stride of the staged B: a fragment's 4 k on different banks
__host__ __device__ constexpr int narrow_ld(int cols) { return ((cols + 7) & ~7) + 4; }
constexpr int NR_BUF = 512;       // elements of a warp's A buffer: its rows times 16 k (32 rows) or 64 k (8 rows)
constexpr int NR_AMAX = 16;       // A blocks of a chunk staged in shared memory, at most
constexpr int NR_WARPS = 4;
constexpr int NR_THREADS = 32 * NR_WARPS;

struct NrChunk {
  int32_t a_begin, a_end;  // its A blocks in nr_a
  int32_t ktot;            // and the k of all of them
  int32_t b_begin, b_end;  // its B blocks in nr_b
  int32_t c_begin, cols;   // its columns in nr_c
  int32_t m;               // rows (shared by its output blocks)
  int32_t d0;              // row r = r0 + d0 r1; 0: rows through the offset tables
};
struct NrTask {            // some rows of a chunk
  NrChunk ch;
  int32_t row0, tiles, pad;  // first row, and its rows in tiles of RW x NR_WARPS
};
struct NrA {               // an A block of a chunk: element (row (r0, r1), k) at off + r0 s0 + r1 s1 + k ks
  int64_t off;
  int32_t s0, s1;          // d0 == 0: s0 is the row table
  int32_t k0, k;           // its first k in the chunk, and how many
  int32_t ks, pad;
};
struct NrB {               // one B block of a chunk: element (k, column) at off + k ks + column cs (or the tables)
  int64_t off;
  int32_t k0, c0;          // its first k and column in the chunk
  int32_t k, n, ks, cs, ktab, ctab;
};

__device__ __forceinline__ void dmma_k4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// elements of one A buffer for chunks of at most ktot k: whole, or NR_BUF at a time
__host__ __device__ constexpr int narrow_buf(int ktot, int rw) {
  return rw * ((ktot + 3) & ~3) < NR_BUF ? rw * ((ktot + 3) & ~3) : NR_BUF;
}
__host__ __device__ constexpr size_t narrow_smem(int ktot, int rw, int ld) {
  return sizeof(double) * ((size_t)NR_WARPS * 2 * narrow_buf(ktot, rw) + (size_t)((ktot + 3) & ~3) * ld);
}

// The B blocks of a chunk, its k from s0 to s1, into shared memory (row stride ld): a
// warp per block, 8 k x 4 columns at a time.  first: the warp's first block, fetched
// before.  Asynchronous copies, which the caller waits for: as loads they came one
// after the other, and 160 k of 16 columns took 20 us.
__device__ __forceinline__ void stage_b(double* sb, int ld, int s0, int s1, const double* B, const NrB* __restrict__ nb,
                                        int b_end, int q, int warps, NrB E, const int32_t* __restrict__ tab) {
  const int lane = threadIdx.x & 31;
  while (q < b_end) {
    const double* Bp = B + E.off;
    const int lo = max(s0 - E.k0, 0), hi = min(s1 - E.k0, E.k);
    for (int c = lane >> 3; c < E.n; c += 4)
      for (int kk = lo + (lane & 7); kk < hi; kk += 8)
        cp_async8(sb + (E.k0 + kk - s0) * ld + E.c0 + c, Bp + (int64_t)(E.ks != NO_STRIDE ? kk * E.ks : tab[E.ktab + kk]) +
                                                             (E.cs != NO_STRIDE ? c * E.cs : tab[E.ctab + c]));
    q += warps;
    if (q < b_end) E = nb[q];
  }
  cp_async_commit();
}

// RW: rows of a warp's tile, 32 or 8
template <int RW>
__global__ void __launch_bounds__(NR_THREADS, 4)
narrow_dgemm(const NrTask* __restrict__ tasks, const NrA* __restrict__ na, const NrB* __restrict__ nb,
             const int64_t* __restrict__ nc, const int32_t* __restrict__ tab, const double* __restrict__ A, const double* __restrict__ B,
             double* __restrict__ C, double alpha, int abuf, int ld, unsigned long long* stamp) {
  extern __shared__ double smem[];
  __shared__ int64_t sc[NR_N];
  __shared__ NrA sa[NR_AMAX];  // the chunk's A blocks, from the second fetch on
  const NrTask task = tasks[blockIdx.x];
  const NrChunk& ch = task.ch;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int ktot = ch.ktot, kz = (ktot + 3) & ~3;
  constexpr int KB = NR_BUF / RW, MT = RW / 8, ROWS = RW * NR_WARPS, LK = 32 / RW;
  double* buf = smem + warp * 2 * abuf;      // this warp's two A buffers, [k][RW rows]
  double* sb = smem + NR_WARPS * 2 * abuf;   // B, [kz][ld]
  // row r of k in a buffer: a fragment's 4 k x 4 rows on different banks
  auto at = [](int k, int r) { return RW * k + (RW == 32 ? r ^ ((k & 3) << 2) : r); };
  const int nblk = ch.a_end - ch.a_begin;
  if (tid < ch.cols) sc[tid] = nc[ch.c_begin + tid];
  if (tid < min(nblk, NR_AMAX)) sa[tid] = na[ch.a_begin + tid];

  // tiles of this warp: rows task.row0 + RW (NR_WARPS i + warp), i < tiles
  const int left = ch.m - task.row0 - RW * warp;
  const int tiles = left <= 0 ? 0 : min(task.tiles, (left + ROWS - 1) / ROWS);
  const int nkb = (ktot + KB - 1) / KB;
  auto row_of = [&](int tile) { return task.row0 + RW * (NR_WARPS * tile + warp); };
  // copies k [KB kb, ...) of a tile into buffer b; lanes past the last row repeat it
  const NrA* blocks = na + ch.a_begin;
  auto fetch = [&](int tile, int kb, int b) {
    const int row = lane % RW, sub = lane / RW;  // LK k at a time
    const int r = min(row_of(tile) + row, ch.m - 1);
    const int r1 = ch.d0 != 0 ? r / ch.d0 : 0, r0 = r - r1 * ch.d0;
    const int klo = kb * KB, khi = min(klo + KB, ktot);
    double* dst = buf + b * abuf;
    for (int q = 0; q < nblk; ++q) {
      const NrA x = blocks[q];
      const int lo = max(klo, x.k0), hi = min(khi, x.k0 + x.k);
      if (lo >= hi) continue;
      const double* p = A + x.off + (int64_t)(lo + sub - x.k0) * x.ks + (ch.d0 != 0 ? r0 * x.s0 + r1 * x.s1 : tab[x.s0 + r]);
#pragma unroll 4
      for (int k = lo - klo + sub; k < hi - klo; k += LK) {
        cp_async8(dst + at(k, row), p);
        p += LK * x.ks;
      }
    }
    const int kend = khi - klo;
    for (int k = kend + sub; k < ((kend + 3) & ~3); k += LK) dst[at(k, row)] = 0.0;
  };
  int q = ch.b_begin + warp;
  NrB E;
  if (q < ch.b_end) E = nb[q];
  after_previous(tab, stamp);
  asm volatile("" : "+l"(B) : : "memory");
  // the chunk's B, and behind it the first k of A; zero where there is no column or k
  stage_b(sb, ld, 0, ktot, B, nb, ch.b_end, q, NR_WARPS, E, tab);
  if (tiles > 0 && nkb > 0) fetch(0, 0, 0);
  cp_async_commit();
  if (tid < (kz - ktot) * ld) sb[ktot * ld + tid] = 0.0;
  const int cpad = ch.cols + (lane & 7);
  if (cpad < ((ch.cols + 7) & ~7))
    for (int k = 4 * warp + (lane >> 3); k < ktot; k += 4 * NR_WARPS) sb[k * ld + cpad] = 0.0;
  cp_async_wait<1>();
  __syncthreads();
  if (nblk <= NR_AMAX) blocks = sa;

  const int nt = (ch.cols + 7) >> 3;  // 8-column parts
  int b = 0;
  for (int tile = 0; tile < tiles; ++tile) {
    double acc[MT][4][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    for (int kb = 0; kb < nkb; ++kb, b ^= 1) {
      if (kb + 1 < nkb) fetch(tile, kb + 1, b ^ 1);
      else if (tile + 1 < tiles) fetch(tile + 1, 0, b ^ 1);
      cp_async_commit();
      cp_async_wait<1>();
      __syncwarp();
      const int kn = min(KB, ktot - kb * KB);
      const double* as = buf + b * abuf;
      const double* bs = sb + (kb * KB + t4) * ld + g;
#pragma unroll 2
      for (int k = 0; k < kn; k += 4) {
        double a[MT];
#pragma unroll
        for (int i = 0; i < MT; ++i) a[i] = as[at(k + t4, 8 * i + g)];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j < nt) {
            const double bv = bs[k * ld + 8 * j];
#pragma unroll
            for (int i = 0; i < MT; ++i) dmma_k4(acc[i][j], a[i], bv);
          }
        }
      }
      __syncwarp();  // the buffer is free for the fetch after next
    }
    const int r = row_of(tile) + g;
    const bool inside = row_of(tile) + RW <= ch.m;
    if (alpha != 1.0) {
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j][0] *= alpha;
          acc[i][j][1] *= alpha;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * j + 2 * t4 + e;
        if (c >= ch.cols) continue;
        double* p = C + sc[c] + r;
        if (inside) {
#pragma unroll
          for (int i = 0; i < MT; ++i) p[8 * i] = acc[i][j][e];
        } else {
#pragma unroll
          for (int i = 0; i < MT; ++i)
            if (r + 8 * i < ch.m) p[8 * i] = acc[i][j][e];
        }
      }
  }
  cp_async_wait<0>();
}

// The same chunks with a thread per row, its up to NC columns as FP64 sums in registers,
// 16 loads of A in flight: no fragment is padded and A does not pass through shared
// memory.  Better where a chunk has few columns, which is where the products above are
// mostly padding and instruction issue (1e6 rows, k = 160: 1 column 190 us, 8 columns
// 238, by fragments 521 and 529; the rule is at the plan).  B is staged whole or, beyond
// RD_SEG bytes, in segments of kseg k, anew for every tile.
constexpr int RD_COLS = 16;            // columns of a chunk, at most
constexpr int RD_SEG = 96 * 1024;      // bytes of staged B, at most

// SEG: more k than a segment, 256 rows to a CTA, else 128.  Block (x, y) has tile y of
// task x.
template <int NC, bool SEG>
__global__ void __launch_bounds__(SEG ? 256 : 128)
rows_dgemm(const NrTask* __restrict__ tasks, const NrA* __restrict__ na, const NrB* __restrict__ nb,
           const int64_t* __restrict__ nc, const int32_t* __restrict__ tab, const double* __restrict__ A,
           const double* __restrict__ B, double* __restrict__ C, double alpha, int kseg, unsigned long long* stamp) {
  extern __shared__ double smem[];  // B, [kseg][NC]
  __shared__ int64_t sc[NC];
  __shared__ NrA sa[NR_AMAX];
  const NrTask task = tasks[blockIdx.x];
  const NrChunk& ch = task.ch;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int nblk = ch.a_end - ch.a_begin, ktot = ch.ktot;
  const int row = task.row0 + (int)(blockDim.x * blockIdx.y) + tid, r = min(row, ch.m - 1);
  if (tid < ch.cols) sc[tid] = nc[ch.c_begin + tid];
  if (tid < min(nblk, NR_AMAX)) sa[tid] = na[ch.a_begin + tid];
  const NrA* blocks = nblk <= NR_AMAX ? sa : na + ch.a_begin;
  after_previous(tab, blockIdx.y == 0 ? stamp : nullptr);
  if ((int)blockIdx.y >= task.tiles) return;
  asm volatile("" : "+l"(A), "+l"(B) : : "memory");
  auto stage = [&](int s0, int s1) {
    const int q0 = ch.b_begin + warp;
    NrB E;
    if (q0 < ch.b_end) E = nb[q0];
    stage_b(smem, NC, s0, s1, B, nb, ch.b_end, q0, blockDim.x >> 5, E, tab);
    cp_async_wait<0>();
    __syncthreads();
  };
  if (!SEG || ktot == 0) stage(0, ktot);
  const int r1 = ch.d0 != 0 ? r / ch.d0 : 0, r0 = r - r1 * ch.d0;
  double acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = 0.0;
  // n k at a time, their loads in flight together
  auto run = [&](auto n, int& k, int hi, const double*& p, const double*& w, int32_t ks) {
    constexpr int U = decltype(n)::value;
    for (; k + U <= hi; k += U) {
      double a[U];
#pragma unroll
      for (int u = 0; u < U; ++u) a[u] = p[(int64_t)u * ks];
      p += (int64_t)U * ks;
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] = fma(a[u], w[c], acc[c]);
        w += NC;
      }
    }
  };
  auto add = [&](const NrA& x, int s0, int s1) {
    int k = max(s0, x.k0);
    const int hi = min(s1, x.k0 + x.k);
    const double* p = A + x.off + (int64_t)(k - x.k0) * x.ks + (ch.d0 != 0 ? r0 * x.s0 + r1 * x.s1 : tab[x.s0 + r]);
    const double* w = smem + (k - s0) * NC;
    run(std::integral_constant<int, 16>(), k, hi, p, w, x.ks);
    run(std::integral_constant<int, 8>(), k, hi, p, w, x.ks);
    run(std::integral_constant<int, 4>(), k, hi, p, w, x.ks);
    run(std::integral_constant<int, 2>(), k, hi, p, w, x.ks);
    run(std::integral_constant<int, 1>(), k, hi, p, w, x.ks);
  };
  if (!SEG) {
    for (int q = 0; q < nblk; ++q) add(blocks[q], 0, ktot);
  } else {
    int q = 0;  // the A block that holds the next k
    for (int s0 = 0; s0 < ktot; s0 += kseg) {
      const int s1 = min(s0 + kseg, ktot);
      if (s0 > 0) __syncthreads();  // the segment before is read
      stage(s0, s1);
      for (; q < nblk; ++q) {
        const NrA x = blocks[q];
        add(x, s0, s1);
        if (x.k0 + x.k > s1) break;  // the rest of its k is in the next segment
      }
    }
  }
  if (row >= ch.m) return;
#pragma unroll
  for (int c = 0; c < NC; ++c)
    if (c < ch.cols) C[sc[c] + row] = alpha * acc[c];
}

// ---------------------------------------------------------------------------
// Mixed-precision path: tcgen05 (5th-generation tensor cores), kind::tf32.
//
// Two launches per contraction.  pack_tf32_ab converts every operand block
// once into TF32 hi/lo tiles (x = hi + lo, both rounded to nearest) stored in
// the exact K-major 128-byte-swizzled layout of a shared-memory MMA operand
// tile; grouped_tc_persist then feeds the tensor cores from those tiles with
// bulk copies and accumulates 128 x 128 output tiles in tensor memory (FP32).
// The split form issues hi*hi + hi*lo + lo*hi per k-step.
constexpr int TC_BM = 128;
constexpr int TC_BN = 128;
constexpr int TC_BK = 32;                        // fp32 elements = one 128-byte swizzle row
constexpr uint32_t TC_WAIT_LIMIT = 1u << 26;
static_assert(TC_BN == TC_BM, "packed tiles are 128 rows for both operands");

// Instruction descriptor: D f32, A/B tf32, both K-major, N = TC_BN, M = TC_BM.
constexpr uint32_t TC_IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TC_BN >> 3) << 17) |
                              ((uint32_t)(TC_BM >> 4) << 24);

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor, K-major with 128-byte swizzle: rows of 128
// bytes, 8-row groups 1024 bytes apart (stride byte offset), version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;              // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset
  d |= (uint64_t)1 << 46;              // descriptor version
  d |= (uint64_t)2 << 61;              // SWIZZLE_128B
  return d;
}

// Byte offset of element (row r, k) in a K-major 128B-swizzled tile.
__device__ __forceinline__ uint32_t sw128_off(int r, int k) {
  return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((((k >> 2) ^ (r & 7))) << 4) + (k & 3) * 4);
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void mbar_init(uint32_t addr, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t addr, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(addr), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait for the phase with the given parity; false on timeout
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t addr, uint32_t parity, uint32_t limit = TC_WAIT_LIMIT) {
  for (uint32_t it = 0; it < limit; ++it)
    if (mbar_try_wait(addr, parity)) return true;
  return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %3, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %4, p;\n\t}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(accumulate), "r"(TC_IDESC)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// ---- operand packing: FP64 blocks -> TF32 hi/lo tiles, pre-swizzled --------
// A packed tile holds 128 rows x 32 k of one operand block as TF32 hi
// (16 KB) followed by TF32 lo (16 KB), each laid out exactly as the K-major
// 128-byte-swizzled shared-memory tile the MMA reads, so one bulk copy moves
// it into shared memory unchanged.  Edges are zero-padded.  Tile (rt, kt) of
// a block sits at base + (rt * kt_count + kt) * 32 KB.
struct PackJob {
  int64_t x_off;             // block offset in the operand (elements)
  int64_t dst;               // packed block base (bytes)
  int32_t rows, K;           // logical rows (m or n) and k
  int32_t row_tab, k_tab;    // offset tables: element = X[x_off + tab[row_tab + r] + tab[k_tab + k]]
  int32_t kt_count;
  int32_t row_unit;          // rows have unit stride: walk them fastest
};
struct PackTile {
  int32_t job, rt, kt;
};
constexpr int TC_TILE_BYTES = 2 * TC_BM * TC_BK * 4;  // hi + lo = 32 KB

// ---- grouped tcgen05 GEMM over packed tiles ---------------------------------
// A block pair in packed form: the bases of its A and B packed blocks and its
// number of 32-wide k-chunks.  The GEMM kernel (grouped_tc_persist below)
// streams each chunk's A and B tiles into a TC_RING-stage ring of
// TC_RING_STAGE bytes with plain bulk copies.
struct PairTC {
  int64_t a_base, b_base;  // packed block bases (bytes)
  int32_t kt;              // k tiles of the pair
  int32_t pad;
};
constexpr int TC_RING = 3;
constexpr int TC_RING_STAGE = 4 * TC_BM * TC_BK * 4;  // A hi, A lo, B hi, B lo: 64 KB
constexpr size_t TC_BULK_SMEM = (size_t)TC_RING * TC_RING_STAGE + 1024;

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}

// ---- persistent form --------------------------------------------------------
// One CTA per SM walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// (longest first) with specialised warps: warp 0 (one thread) streams the
// packed tiles of every k-chunk of every tile into the TC_RING-stage ring,
// running ahead across tile boundaries; warp 1 (one thread) issues the MMAs
// into one of two 128-column TMEM accumulators, alternating per tile, and
// commits each stage to its empty barrier and each finished tile to the
// accumulator's full barrier; warps 2-5 drain a finished accumulator
// (tcgen05.ld, alpha * acc as FP64) while the MMAs of the next tile fill the
// other one, then release it through the accumulator's empty barrier (four
// arrivals).  A warp may read only its quarter of the 128 TMEM lanes (warp
// index mod 4), so warps 2, 3, 4, 5 cover lanes 64, 96, 0, 32.  Every wait is
// bounded; on timeout the CTA records TT_ERR_TIMEOUT, stops issuing, lets
// what it issued land (bounded) and frees TMEM.
constexpr int TC_P_THREADS = 192;
constexpr uint32_t TC_P_COLS = 2 * TC_BN;

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

template <bool SPLIT>
__global__ void __launch_bounds__(TC_P_THREADS, 1)
grouped_tc_persist(const TaskDev* __restrict__ tasks, int n_tasks, const OutDev* __restrict__ outs,
                   const PairTC* __restrict__ pairs, const uint8_t* __restrict__ packA,
                   const uint8_t* __restrict__ packB, double* __restrict__ C, double alpha, int* __restrict__ status,
                   int* __restrict__ ctx_status, uint32_t wait_limit) {
  extern __shared__ uint8_t tc_smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[TC_RING], empty_bar[TC_RING], accf_bar[2], acce_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int flag;
  __shared__ int issued, consumed, committed_tiles;

  const uint32_t sbase = (smem_u32(tc_smem_raw) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t half = SPLIT ? (uint32_t)TC_TILE_BYTES : (uint32_t)(TC_TILE_BYTES / 2);  // bytes per operand tile

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TC_P_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < TC_RING; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&accf_bar[b]), 1);
      mbar_init(smem_u32(&acce_bar[b]), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    flag = 0;
    issued = 0;
    consumed = 0;
    committed_tiles = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {  // producer
      int g = 0;
      for (int t = blockIdx.x; t < n_tasks && !flag; t += gridDim.x) {
        const TaskDev task = tasks[t];
        const int rt = task.m0 / TC_BM, nt = task.n0 / TC_BN;
        for (int p = task.p_begin; p < task.p_end && !flag; ++p) {
          const PairTC q = pairs[p];
          for (int kt = 0; kt < q.kt; ++kt, ++g) {
            const int s = g % TC_RING;
            if (g >= TC_RING &&
                !mbar_wait_bounded(smem_u32(&empty_bar[s]), (uint32_t)((g / TC_RING - 1) & 1), wait_limit)) {
              flag = 1;
              break;
            }
            const uint32_t st = sbase + s * TC_RING_STAGE;
            mbar_expect_tx(smem_u32(&full_bar[s]), 2 * half);
            bulk_g2s(st, packA + q.a_base + (int64_t)(rt * q.kt + kt) * TC_TILE_BYTES, half, smem_u32(&full_bar[s]));
            bulk_g2s(st + TC_TILE_BYTES, packB + q.b_base + (int64_t)(nt * q.kt + kt) * TC_TILE_BYTES, half,
                     smem_u32(&full_bar[s]));
            issued = g + 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      int g = 0, i = 0;
      for (int t = blockIdx.x; t < n_tasks && !flag; t += gridDim.x, ++i) {
        const TaskDev task = tasks[t];
        int nch = 0;
        for (int p = task.p_begin; p < task.p_end; ++p) nch += pairs[p].kt;
        const int b = i & 1;
        if (i >= 2 && !mbar_wait_bounded(smem_u32(&acce_bar[b]), (uint32_t)(((i >> 1) - 1) & 1), wait_limit)) {
          flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t acc_tm = tmem + (uint32_t)(b * TC_BN);
        for (int c = 0; c < nch; ++c, ++g) {
          const int s = g % TC_RING;
          if (!mbar_wait_bounded(smem_u32(&full_bar[s]), (uint32_t)((g / TC_RING) & 1), wait_limit)) {
            flag = 1;
            break;
          }
          tc_fence_after();
          const uint32_t ah = sbase + s * TC_RING_STAGE, al = ah + TC_TILE_BYTES / 2;
          const uint32_t bh = ah + TC_TILE_BYTES, bl = bh + TC_TILE_BYTES / 2;
#pragma unroll
          for (int kk = 0; kk < TC_BK / 8; ++kk) {
            const uint32_t adv = 32u * kk;
            const uint32_t acc = (c > 0 || kk > 0) ? 1u : 0u;
            if (SPLIT) {
              mma_tf32(acc_tm, sw128_desc(al + adv), sw128_desc(bh + adv), acc);
              mma_tf32(acc_tm, sw128_desc(ah + adv), sw128_desc(bl + adv), 1u);
              mma_tf32(acc_tm, sw128_desc(ah + adv), sw128_desc(bh + adv), 1u);
            } else {
              mma_tf32(acc_tm, sw128_desc(ah + adv), sw128_desc(bh + adv), acc);
            }
          }
          mma_commit(smem_u32(&empty_bar[s]));
          consumed = g + 1;
        }
        if (flag) break;
        if (nch > 0) mma_commit(smem_u32(&accf_bar[b]));
        else mbar_arrive(smem_u32(&accf_bar[b]));
        committed_tiles = i + 1;
      }
    }
  } else {  // epilogue, warps 2..5
    const int q4 = warp & 3;
    int i = 0;
    for (int t = blockIdx.x; t < n_tasks; t += gridDim.x, ++i) {
      // decisions are warp-uniform: the TMEM loads below are .sync.aligned
      if (__any_sync(0xffffffffu, flag != 0)) break;
      const TaskDev task = tasks[t];
      const OutDev out = outs[task.out];
      int nch = 0;
      for (int p = task.p_begin; p < task.p_end; ++p) nch += pairs[p].kt;
      const int b = i & 1;
      const bool ok = mbar_wait_bounded(smem_u32(&accf_bar[b]), (uint32_t)((i >> 1) & 1), wait_limit);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) flag = 1;
        break;
      }
      tc_fence_after();
      double* Cb = C + out.c_off;
      const int m = task.m0 + q4 * 32 + lane;
#pragma unroll
      for (int c16 = 0; c16 < TC_BN / 16; ++c16) {
        float v[16];
        if (nch > 0) {
          tmem_ld16(tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(b * TC_BN + c16 * 16), v);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = 0.f;
        }
        if (m < out.m) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int n = task.n0 + c16 * 16 + j;
            if (n < out.n) Cb[m + (int64_t)out.ldc * n] = alpha * (double)v[j];
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acce_bar[b]));
    }
  }
  __syncwarp();
  __syncthreads();
  if (tid == 0 && flag) {
    // let the copies that were issued but not consumed land and the last
    // committed MMAs finish before shared and tensor memory are released
    for (int g = consumed; g < issued; ++g)
      mbar_wait_bounded(smem_u32(&full_bar[g % TC_RING]), (uint32_t)((g / TC_RING) & 1));
    if (consumed > 0)
      mbar_wait_bounded(smem_u32(&empty_bar[(consumed - 1) % TC_RING]), (uint32_t)(((consumed - 1) / TC_RING) & 1));
    if (committed_tiles > 0) {  // the last tile commit's arrival
      const int il = committed_tiles - 1;
      mbar_wait_bounded(smem_u32(&accf_bar[il & 1]), (uint32_t)((il >> 1) & 1));
    }
    atomicExch(status, TT_ERR_TIMEOUT);
    atomicExch_system(ctx_status, TT_ERR_TIMEOUT);  // the context's mapped status word
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_P_COLS) : "memory");
}

// Both operands' packing in one launch: tiles [0, n_a) of A, then those of B.
template <bool SPLIT>
__global__ void __launch_bounds__(128)
pack_tf32_ab(const PackJob* __restrict__ jobsA, const PackTile* __restrict__ tilesA, int n_a,
             const PackJob* __restrict__ jobsB, const PackTile* __restrict__ tilesB, const int32_t* __restrict__ tab,
             const double* __restrict__ A, const double* __restrict__ B, uint8_t* __restrict__ pa,
             uint8_t* __restrict__ pb) {
  // the tile is assembled in shared memory at its swizzled offsets, then
  // written out with consecutive 16-byte stores (a thread's 16 bytes of a
  // row would otherwise land in a different 128-byte line per lane)
  __shared__ __align__(128) uint8_t st[TC_TILE_BYTES];
  const bool is_a = (int)blockIdx.x < n_a;
  const PackTile t = is_a ? tilesA[blockIdx.x] : tilesB[blockIdx.x - n_a];
  const PackJob J = is_a ? jobsA[t.job] : jobsB[t.job];
  const double* X = is_a ? A : B;
  const int tid = threadIdx.x;
  uint8_t* dst = (is_a ? pa : pb) + J.dst + (int64_t)(t.rt * J.kt_count + t.kt) * TC_TILE_BYTES;
  if (J.row_unit) {  // rows are contiguous: a thread has a row, four k at a time
    const int gr = t.rt * TC_BM + tid, row = gr < J.rows ? tab[J.row_tab + gr] : 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      double x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gk = t.kt * TC_BK + 4 * i + e;
        x[e] = (gr < J.rows && gk < J.K) ? X[J.x_off + row + tab[J.k_tab + gk]] : 0.0;
      }
      uint32_t h[4], l[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        h[e] = to_tf32(__double2float_rn(x[e]));
        l[e] = SPLIT ? to_tf32(__double2float_rn(x[e] - (double)__uint_as_float(h[e]))) : 0u;
      }
      const uint32_t o = sw128_off(tid, 4 * i);
      *reinterpret_cast<uint4*>(st + o) = make_uint4(h[0], h[1], h[2], h[3]);
      if (SPLIT) *reinterpret_cast<uint4*>(st + TC_TILE_BYTES / 2 + o) = make_uint4(l[0], l[1], l[2], l[3]);
    }
  } else {
    // a warp has a row, a lane a k: 256 contiguous bytes a load where k is contiguous
    // (eight lanes per row with four k each took four passes over the same sectors:
    // five products at m = 717 1121 us, now 1050; at m = 3072 16.1 ms, now 15.5)
    const int lane = tid & 31, gk = t.kt * TC_BK + lane, col = gk < J.K ? tab[J.k_tab + gk] : 0;
#pragma unroll 16
    for (int i = 0; i < TC_BM / 4; ++i) {
      const int r = (tid >> 5) + 4 * i, gr = t.rt * TC_BM + r;
      const double x = (gr < J.rows && gk < J.K) ? X[J.x_off + tab[J.row_tab + gr] + col] : 0.0;
      const uint32_t h = to_tf32(__double2float_rn(x));
      const uint32_t o = sw128_off(r, lane & ~3) + 4 * (lane & 3);
      *reinterpret_cast<uint32_t*>(st + o) = h;
      if (SPLIT)
        *reinterpret_cast<uint32_t*>(st + TC_TILE_BYTES / 2 + o) = to_tf32(__double2float_rn(x - (double)__uint_as_float(h)));
    }
  }
  __syncthreads();
  constexpr int NV = (SPLIT ? TC_TILE_BYTES : TC_TILE_BYTES / 2) / 16;
#pragma unroll 4
  for (int v = tid; v < NV; v += blockDim.x)
    reinterpret_cast<uint4*>(dst)[v] = reinterpret_cast<const uint4*>(st)[v];
}

// CTAs that share a tile's k range in grouped_dgemm, for plans of `tiles` tiles of at
// most `longest` chunks.  While there are fewer than two CTAs per SM, each keeps two
// chunks of the longest tile; a long k is shared also while there are fewer than two
// rounds (four CTAs fit an SM) and each keeps 12.  R at bond dimension 1400 (420 tiles, k
// up to 6552): 1110 us whole, 730 in four; stopping at one round 860.  The products of a
// chain at 128 (34 tiles of at most 12 chunks): 129 us per three products whole, 123 down
// to four chunks, 105 down to two.  Two chunks up to two rounds paid more for the
// exchange than for the idle SMs: environment update of the cylinder at 400 85 us, now
// 67, at 700 190 and 155; with 8 chunks instead of 12 a chain's at 957 130, now 120, with
// 16 three products of a chain at 700 350, now 296.
int dgemm_split(int64_t tiles, int longest, int num_sms) {
  int split = 1;
  while (split < SPLIT_MAX && ((tiles * split < 2 * (int64_t)num_sms && longest / (2 * split) >= 2) ||
                               (tiles * split < 8 * (int64_t)num_sms && longest / (2 * split) >= 12)))
    split *= 2;
  return split;
}

// Cost model of the *_AUTO precisions: predicted device time (microseconds) of one exec
// of a contraction in `prec` (FP64, or a tcgen05 kind with its two packing launches).
// Fitted to 242 contractions (1 to 40 blocks of 40 x 40 to 20000 x 40, k of 64 to 6000, and
// blocks of mixed sizes as a bond has): FP64 0.79 to 1.15 and 3xTF32 0.77 to 1.02 of the
// measured time (tenth to ninetieth per cent).  The choice that it leads to cost more than
// 1.15 of the better one in 8 of them, at most 1.41, all but one by staying in FP64.
//   FP64 tiles: c CTAs of an SM take 0.6 + 0.58 c us per chunk of 16 k together (1.2 us
//     alone, the latencies of one chunk; 0.73 each where four share the SM), a tile 1.5
//     chunks more for its start and end; CTAs come in rounds of four per SM, and a tile's k
//     range is shared as the plan shares it.
//   FP64 narrow chunks: bound by their bytes.
//   Tensor cores: 0.57 us per chunk of 32 k and tile in 3xTF32, a tile at a time per SM;
//     the packed operands and C pass through memory, and before that every operand is read
//     and written packed (kept operands once for kKeptUses execs).
double predict_us(const tt_out_block* outs, int n_out, const std::vector<PairDev>& hp,
                  const std::vector<int>& first, int prec, int num_sms, int keep = 0) {
  constexpr double kHbm = 5.0e6, kKeptUses = 4.0;  // bytes per us
  const double sms = std::max(1, num_sms);
  const bool tc = prec != TT_PREC_FP64;
  const int tm = tc ? TC_BM : BM, tn = tc ? TC_BN : BN;
  auto up = [](int x, int t) { return (double)((x + t - 1) / t) * t; };
  // a pair's k in chunks: of 32, or of 16, whose last one costs less where 8 or fewer are left
  auto cost = [&](int k) { return tc ? up(k, TC_BK) / TC_BK : k / BK + (k % BK == 0 ? 0.0 : k % BK <= 8 ? 0.7 : 1.0); };
  double tiles = 0.0, total = 0.0, longest = 0.0, c_bytes = 0.0;
  int chunks = 0;  // of the longest tile, as the plan counts them
  bool narrow = !tc;
  std::map<int64_t, std::pair<double, double>> ua, ub;  // distinct operand blocks: (elements, padded elements)
  for (int o = 0; o < n_out; ++o) {
    double task = 0.0;
    int whole = 0;
    int64_t k = 0;
    for (int i = first[o]; i < first[o + 1]; ++i) {
      const PairDev& P = hp[i];
      task += cost(P.k);
      whole += (P.k + BK - 1) / BK;
      k += P.k;
      narrow = narrow && P.k <= NR_K;
      ua.emplace(P.a_off, std::make_pair((double)P.m * P.k, up(P.m, tm) * up(P.k, TC_BK)));
      ub.emplace(P.b_off, std::make_pair((double)P.n * P.k, up(P.n, tn) * up(P.k, TC_BK)));
    }
    narrow = narrow && outs[o].n <= NR_N && k <= NR_KTOT;
    const double t = up(outs[o].m, tm) / tm * (up(outs[o].n, tn) / tn);
    tiles += t;
    total += t * task;
    if (t > 0) {
      longest = std::max(longest, task);
      chunks = std::max(chunks, whole);
    }
    c_bytes += 8.0 * outs[o].m * outs[o].n;
  }
  double read = 0.0, pack = 0.0, packed = 0.0;
  const double per = prec == TT_PREC_TF32X3 ? 8.0 : 4.0;  // bytes of a packed element
  for (int w = 0; w < 2; ++w) {
    const double share = ((keep >> w) & 1) ? 1.0 / kKeptUses : 1.0;
    for (const auto& kv : (w == 0 ? ua : ub)) {
      read += 8.0 * kv.second.first;
      pack += (8.0 * kv.second.first + per * kv.second.second) * share;
      packed += per * kv.second.second;
    }
  }
  if (narrow) return 3.0 + (read + c_bytes) / 3.0e6;
  if (tc) {
    const double tau = prec == TT_PREC_TF32X3 ? 0.57 : 0.25;
    const double rounds = tiles <= 4 * sms ? std::ceil(tiles / sms) : tiles / sms;
    const double mma = std::max(longest, tiles > 0 ? rounds * total / tiles : 0.0) * tau;
    return 12.0 + pack / kHbm + std::max(mma, (packed + c_bytes) / kHbm);
  }
  const int split = dgemm_split((int64_t)tiles, chunks, num_sms);
  const double ctas = tiles * split, avg = ctas > 0 ? total / ctas + 1.5 : 0.0;
  auto tau = [](double c) { return c > 0 ? 0.6 + 0.58 * c : 0.0; };  // c CTAs of an SM, a chunk each
  const double full = std::floor(ctas / (4 * sms)), rest = std::ceil((ctas - full * 4 * sms) / sms);
  const double math = std::max((longest / split + 1.5) * tau(1), avg * (full * tau(4) + tau(rest)));
  return 2.5 + (split > 1 ? 1.5 : 0.0) + std::max(math, (read + c_bytes) / 6.0e6);
}

}  // namespace

struct tt_plan {
  int precision = TT_PREC_FP64;
  char* d_blob = nullptr;  // the device buffer that every array below lies in
  // narrow FP64 plans (narrow_dgemm)
  bool narrow = false;
  int nr_ktot = 0;  // the most k of a chunk
  int nr_rw = 32;   // rows of a warp's tile
  int nr_cols = 0;  // the most columns of a chunk
  int rd_threads = 0;  // rows_dgemm in its place: rows of a CTA,
  int rd_tiles = 1;    // and its tiles of a task, at most
  NrTask* d_nr_tasks = nullptr;
  NrA* d_nr_a = nullptr;
  NrB* d_nr_b = nullptr;
  int64_t* d_nr_c = nullptr;
  int* d_status = nullptr;  // tensor-core path: TT_OK or TT_ERR_TIMEOUT
  // tensor-core path: packing jobs and tiles of the unique A / B blocks, the
  // pairs in packed form, and the packed sizes (buffers are taken from the
  // stream-ordered pool for each exec)
  PackJob* d_jobsA = nullptr;
  PackJob* d_jobsB = nullptr;
  PackTile* d_tilesA = nullptr;
  PackTile* d_tilesB = nullptr;
  PairTC* d_pairtc = nullptr;
  int n_tilesA = 0, n_tilesB = 0;
  int64_t bytesA = 0, bytesB = 0;
  int n_tasks = 0;
  int split = 1;            // grouped_dgemm: CTAs per output tile
  int n_pairs = 0;
  int n_out = 0;
  double flops = 0.0;
  int64_t dev_bytes = 0;  // device memory the plan holds (tables, tasks, packing jobs)
  // tensor-core path: packed operands kept between execs (tt_contract_exec_keep)
  // and the operand each was packed from; released by tt_plan_release_packed
  mutable uint8_t* kept[2] = {nullptr, nullptr};
  mutable const double* kept_src[2] = {nullptr, nullptr};
  // packing buffers reused across execs for operands packed afresh each time
  // (keep bits 2 and 3), so that a run of execs allocates them once
  mutable uint8_t* scratch[2] = {nullptr, nullptr};
  TaskDev* d_tasks = nullptr;
  DTask* d_dtasks = nullptr;  // grouped_dgemm plans, in place of d_tasks
  OutDev* d_outs = nullptr;
  PairDev* d_pairs = nullptr;
  int32_t* d_tab = nullptr;
};

extern "C" {

// Host seconds of the planner's stages on this thread (tt_contract_plan_timers):
// pair tables, precision choice, tile tasks and the narrow chunks,
// tensor-core packing jobs, device tables and uploads.
static thread_local double g_plan_stage_s[5];
struct PlanLap {
  std::chrono::steady_clock::time_point t = std::chrono::steady_clock::now();
  int stage = 0;
  void operator()(int k) {
    const auto now = std::chrono::steady_clock::now();
    g_plan_stage_s[k] += std::chrono::duration<double>(now - t).count();
    t = now;
    stage = k + 1;
  }
  ~PlanLap() {
    if (stage < 5) (*this)(4);
  }
};

int tt_contract_plan(tt_ctx* ctx, const tt_out_block* outs, int n_out,
                     const tt_block_pair* pairs, int n_pairs, int precision,
                     tt_plan** plan_out) {
  return tt_contract_plan_keep(ctx, outs, n_out, pairs, n_pairs, precision, 0, plan_out);
}

int tt_contract_plan_keep(tt_ctx* ctx, const tt_out_block* outs, int n_out, const tt_block_pair* pairs,
                          int n_pairs, int precision, int keep, tt_plan** plan_out) {
  PlanLap lap;
  TT_REQUIRE(ctx && plan_out, "tt_contract_plan: null argument");
  TT_REQUIRE(n_out >= 0 && n_pairs >= 0, "tt_contract_plan: negative count");
  TT_REQUIRE(precision >= TT_PREC_FP64 && precision <= TT_PREC_TF32X3_AUTO,
             "tt_contract_plan: unsupported precision");
  const bool automatic = precision == TT_PREC_TF32_AUTO || precision == TT_PREC_TF32X3_AUTO;
  if (automatic) precision = precision == TT_PREC_TF32_AUTO ? TT_PREC_TF32 : TT_PREC_TF32X3;
  *plan_out = nullptr;
  // pairs grouped by output block (stable: keeps the reference's accumulation order)
  std::vector<int> order(n_pairs);
  std::iota(order.begin(), order.end(), 0);
  for (int i = 0; i < n_pairs; ++i)
    TT_REQUIRE(pairs[i].out_block >= 0 && pairs[i].out_block < n_out,
               "tt_contract_plan: pair references a missing output block");
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return pairs[a].out_block < pairs[b].out_block; });
  std::vector<PairDev> hp(n_pairs);
  std::vector<TableJob> jobs;
  jobs.reserve(4 * (size_t)n_pairs);
  int64_t tab_len = 0;
  std::map<std::vector<int64_t>, int32_t> tab_of;  // table contents -> its number in jobs
  std::vector<int64_t> tab_key;
  double flops = 0.0;
  std::vector<int> first(n_out + 1, 0);
  std::vector<int64_t> work(n_out, 0);
  std::vector<int> chunks(n_out, 0);
  for (int ii = 0; ii < n_pairs; ++ii) {
    const tt_block_pair& q = pairs[order[ii]];
    TT_REQUIRE(q.n_m >= 0 && q.n_m <= TT_MAX_MODES && q.n_k >= 0 && q.n_k <= TT_MAX_MODES &&
                   q.n_n >= 0 && q.n_n <= TT_MAX_MODES,
               "tt_contract_plan: mode count out of range");
    int64_t m = 1, n = 1, k = 1;
    for (int i = 0; i < q.n_m; ++i) m *= q.m_dims[i];
    for (int i = 0; i < q.n_k; ++i) k *= q.k_dims[i];
    for (int i = 0; i < q.n_n; ++i) n *= q.n_dims[i];
    const tt_out_block& o = outs[q.out_block];
    TT_REQUIRE(m == o.m && n == o.n, "tt_contract_plan: pair shape does not match its output block");
    TT_REQUIRE(m < (1ll << 31) && n < (1ll << 31) && k < (1ll << 31), "tt_contract_plan: block too large");
    PairDev P;
    P.a_off = q.a_off;
    P.b_off = q.b_off;
    P.m = (int)m;
    P.n = (int)n;
    P.k = (int)k;
    // an offset table is a function of (length, dims, strides) alone: pairs
    // that address the same rows or columns of a block share one.  rowA ..
    // colB are table numbers until the path is chosen; only the tables that it
    // reads are then laid out
    auto add_job = [&](int len, int nmodes, const int32_t* dims, const int64_t* strides) {
      tab_key.assign({(int64_t)len, (int64_t)nmodes});
      for (int i = 0; i < nmodes; ++i) {
        tab_key.push_back(dims[i]);
        tab_key.push_back(strides[i]);
      }
      auto hit = tab_of.find(tab_key);
      if (hit != tab_of.end()) return hit->second;
      TableJob J;
      memset(&J, 0, sizeof(J));
      J.dst = -1;
      J.len = len;
      J.nmodes = nmodes;
      for (int i = 0; i < nmodes; ++i) {
        J.dims[i] = dims[i];
        J.strides[i] = strides[i];
      }
      const int32_t id = (int32_t)jobs.size();
      jobs.push_back(J);
      tab_of.emplace(tab_key, id);
      return id;
    };
    P.rowA = add_job((int)m, q.n_m, q.m_dims, q.a_m_stride);
    P.colA = add_job((int)k, q.n_k, q.k_dims, q.a_k_stride);
    P.rowB = add_job((int)k, q.n_k, q.k_dims, q.b_k_stride);
    P.colB = add_job((int)n, q.n_n, q.n_dims, q.b_n_stride);
    // coalescing choice only: walk the operand along its unit-stride mode
    bool a_m_unit = q.n_m > 0 && q.a_m_stride[0] == 1;
    bool a_k_unit = q.n_k > 0 && q.a_k_stride[0] == 1;
    P.a_mfast = (a_m_unit || !a_k_unit) ? 1 : 0;
    bool b_k_unit = q.n_k > 0 && q.b_k_stride[0] == 1;
    P.b_kfast = b_k_unit ? 1 : 0;
    // the one stride that a dimension's modes merge into, where they do
    auto merged = [](int nmodes, const int32_t* dims, const int64_t* strides) {
      int64_t st = 0, next = 0;
      bool any = false;
      for (int i = 0; i < nmodes; ++i) {
        if (dims[i] == 1) continue;
        if (any && strides[i] != next) return NO_STRIDE;
        if (!any) st = strides[i];
        any = true;
        next = strides[i] * dims[i];
      }
      return st >= 0 && st <= INT_MAX ? (int32_t)st : NO_STRIDE;
    };
    P.a_rs = merged(q.n_m, q.m_dims, q.a_m_stride);
    P.a_ks = merged(q.n_k, q.k_dims, q.a_k_stride);
    P.b_ks = merged(q.n_k, q.k_dims, q.b_k_stride);
    P.b_cs = merged(q.n_n, q.n_dims, q.b_n_stride);
    hp[ii] = P;
    first[q.out_block + 1]++;
    work[q.out_block] += k;
    chunks[q.out_block] += (int)((k + BK - 1) / BK);
    flops += 2.0 * (double)m * (double)n * (double)k;
  }
  lap(0);
  for (int o = 0; o < n_out; ++o) first[o + 1] += first[o];
  // FP64 unless the tensor-core form is predicted clearly (20 %) faster: the
  // model is coarse, and FP64 is the more accurate of the two
  if (automatic && predict_us(outs, n_out, hp, first, precision, ctx->num_sms, keep) >
                       0.8 * predict_us(outs, n_out, hp, first, TT_PREC_FP64, ctx->num_sms))
    precision = TT_PREC_FP64;
  lap(1);
  const bool tc = precision != TT_PREC_FP64;
  // FP64 plans whose output blocks are at most NR_N wide and whose pairs
  // contract at most NR_K elements run in chunks, on one of the narrow kernels; those
  // with more than NR_KTOT over a block where they are narrow and many (below)
  bool narrow = !tc && n_pairs > 0;
  int64_t klong = 0, rows128 = 0;  // the most k of a block; the blocks' rows in 128s
  for (int o = 0; o < n_out; ++o) {
    klong = std::max(klong, work[o]);
    rows128 += outs[o].n > 0 ? (outs[o].m + 127) / 128 : 0;
  }
  const int most = klong <= NR_KTOT ? NR_N : RD_COLS;  // columns of a chunk
  for (int o = 0; o < n_out && narrow; ++o) narrow = outs[o].n <= most;
  for (int i = 0; i < n_pairs && narrow; ++i) narrow = hp[i].k <= NR_K;
  if (klong > NR_KTOT) narrow = narrow && rows128 >= ctx->num_sms;
  for (int o = 0; o < n_out; ++o)
    TT_REQUIRE(outs[o].m >= 0 && outs[o].n >= 0 && outs[o].ldc >= outs[o].m,
               "tt_contract_plan: bad output block");
  // tile tasks, longest first (LPT) so heavy blocks start early
  const int tile_m = tc ? TC_BM : BM, tile_n = tc ? TC_BN : BN;
  std::vector<TaskDev> tsorted;
  int nr_rw = 32, nr_cols = 0, rd_threads = 0, rd_tiles = 1;
  std::vector<NrTask> nr_tasks;
  std::vector<NrChunk> nr_chunks;
  std::vector<NrA> nr_a;
  std::vector<NrB> nr_b;
  std::vector<int64_t> nr_c;
  // chunks: output blocks whose pairs read the same A blocks the same way (an offset
  // table stands for its modes and strides), so that every k of a chunk belongs to every
  // one of its columns
  std::map<std::vector<int64_t>, std::vector<int>> by_a;  // (rows, A blocks in order) -> output blocks
  std::vector<std::vector<int>> opairs(narrow ? n_out : 0);  // an output block's pairs in that order
  if (narrow) {
    std::vector<int64_t> sig;
    for (int o = 0; o < n_out; ++o) {
      if (outs[o].m == 0 || outs[o].n == 0) continue;
      std::vector<int>& op = opairs[o];
      for (int i = first[o]; i < first[o + 1]; ++i) op.push_back(i);
      auto key = [&](int i) { return std::make_pair(std::make_pair(hp[i].a_off, hp[i].rowA), std::make_pair(hp[i].colA, hp[i].k)); };
      std::stable_sort(op.begin(), op.end(), [&](int x, int y) { return key(x) < key(y); });
      sig.assign(1, outs[o].m);
      for (int i : op) sig.insert(sig.end(), {hp[i].a_off, hp[i].rowA, hp[i].colA, hp[i].k});
      by_a[sig].push_back(o);
    }
    int64_t all = 0;  // the chunks' rows in 128s
    for (const auto& kv : by_a) {
      int cols = 0;
      for (int o : kv.second) {
        if (cols == 0 || cols + outs[o].n > most) {
          all += (outs[o].m + 127) / 128;
          cols = 0;
        }
        cols += outs[o].n;
        nr_cols = std::max(nr_cols, cols);
      }
    }
    // A thread per row or fragments?  Measured over 1e3 to 1e6 rows (in 128s per SM: 0.05
    // to 50), 1 to 32 columns, k of 5 to 1200, each against both and against 64 x 64 tiles:
    // up to 8 columns a thread per row is better once half of the SMs have rows (30000
    // rows, k = 128, 1 and 8 columns: 7.9 and 10.7 us, fragments 17 and 18; 8000 rows, k =
    // 56: 6.4 and 7.8, fragments 5.6 and 6.2), with k of up to 28 four per SM (three
    // products of a chain, k = 8 over many short chunks, 0.8 to 3.8 of them: 82.5 and 112
    // us, fragments 78.5 and 110, 5.1: 135 and 141); up to 16 columns until the
    // FP64 sums of one row outweigh its loads (16 columns, k = 56: 60000 rows 14.5 and
    // 16.3 us, 250000 54 and 48, 1e6 196 and 149; k = 14: 9.1 and 12.7 at 120000, 72 and
    // 71 at 1e6).  With more k than fragments take, tiles are better while there are few
    // rows (16 columns, k = 640: 30000 rows 134 and 86 us, 250000 494 and 480), unless
    // their pairs' k are mostly padding to 16 (200000 rows, 100 pairs of 6: 455 and 810).
    const int64_t sms = ctx->num_sms;
    int64_t kpad = 0, ksum = 0;
    for (int o = 0; o < n_out; ++o) {
      kpad += (int64_t)chunks[o] * BK;
      ksum += work[o];
    }
    bool per_row;
    if (nr_cols > RD_COLS) per_row = false;
    else if (klong <= 28) per_row = all >= 4 * sms && (nr_cols <= 8 || all < 20 * sms || klong <= 16);
    else if (nr_cols <= 8) per_row = klong <= NR_KTOT ? 2 * all >= sms : all >= sms;
    else if (klong <= NR_KTOT) per_row = all >= sms && all < 20 * sms;
    else per_row = all >= 2 * sms && 5 * kpad >= 7 * ksum;
    if (per_row) rd_threads = klong <= NR_KTOT ? 128 : 256;
    else narrow = klong <= NR_KTOT;
    // Fragments: 8 rows to a warp, all of their k in flight at once, where 32 would leave
    // SMs idle (8000 rows, k = 56, 32 columns: 7.3 and 9.8 us; 30000 rows: 15.0 and 11.9)
    nr_rw = all < sms ? 8 : 32;
  }
  if (!narrow) {
    std::vector<int> oorder(n_out);
    std::iota(oorder.begin(), oorder.end(), 0);
    std::stable_sort(oorder.begin(), oorder.end(), [&](int x, int y) { return work[x] > work[y]; });
    for (int o : oorder)
      for (int m0 = 0; m0 < outs[o].m; m0 += tile_m)
        for (int n0 = 0; n0 < outs[o].n; n0 += tile_n) tsorted.push_back(TaskDev{o, m0, n0, first[o], first[o + 1]});
  } else {
    // the two strides (first extent d0) that a pair's row modes merge into;
    // d0 = 0 when they do not.  One stride alone fits any d0, with s1 = s0 d0.
    struct Rows {
      int64_t d0, s0, s1;
      bool one;
    };
    auto rows_of = [&](int i) {
      const tt_block_pair& q = pairs[order[i]];
      Rows r{1, 0, 0, true};
      int groups = 0;
      int64_t next = 0;
      for (int d = 0; d < q.n_m; ++d) {
        const int64_t e = q.m_dims[d], st = q.a_m_stride[d];
        if (e == 1) continue;
        if (groups > 0 && st == next) {
          if (groups == 1) r.d0 *= e;
        } else if (groups == 0) {
          r.d0 = e;
          r.s0 = st;
          groups = 1;
        } else if (groups == 1) {
          r.s1 = st;
          groups = 2;
        } else {
          return Rows{0, 0, 0, false};
        }
        next = st * e;
      }
      r.one = groups <= 1;
      return r;
    };
    std::vector<std::pair<int64_t, std::vector<int>>> groups;  // the chunks of one signature, and their cost
    for (auto& kv : by_a) {
      const std::vector<int>& os = kv.second;
      std::vector<int> ids;
      int64_t cost = 0;
      for (size_t x = 0; x < os.size();) {
        NrChunk c{(int32_t)nr_a.size(), 0, 0, (int32_t)nr_b.size(), 0, (int32_t)nr_c.size(), 0, outs[os[x]].m, 0};
        size_t y = x;
        for (; y < os.size() && c.cols + outs[os[y]].n <= most; ++y) {
          int32_t k0 = 0;
          for (int i : opairs[os[y]]) {
            const PairDev& P = hp[i];
            nr_b.push_back(NrB{P.b_off, k0, c.cols, P.k, P.n, P.b_ks, P.b_cs, P.rowB, P.colB});
            k0 += hp[i].k;
          }
          for (int n = 0; n < outs[os[y]].n; ++n) nr_c.push_back(outs[os[y]].c_off + (int64_t)outs[os[y]].ldc * n);
          c.cols += outs[os[y]].n;
        }
        c.b_end = (int32_t)nr_b.size();
        const std::vector<int>& op = opairs[os[x]];
        std::vector<Rows> rw;
        int64_t d0 = 0;
        bool two = true;
        for (int i : op) {
          rw.push_back(rows_of(i));
          if (rw.back().d0 == 0) two = false;
          if (!rw.back().one) {
            two = two && (d0 == 0 || d0 == rw.back().d0);
            d0 = rw.back().d0;
          }
        }
        if (d0 == 0) d0 = c.m;
        for (size_t u = 0; u < op.size(); ++u) {
          const int64_t s1 = rw[u].one ? rw[u].s0 * d0 : rw[u].s1;
          two = two && rw[u].s0 >= 0 && rw[u].s0 <= INT_MAX && s1 >= 0 && s1 <= INT_MAX;
        }
        c.d0 = two ? (int32_t)d0 : 0;
        for (size_t u = 0; u < op.size(); ++u) {
          const PairDev& P = hp[op[u]];
          const tt_block_pair& q = pairs[order[op[u]]];
          NrA x{P.a_off, two ? (int32_t)rw[u].s0 : P.rowA, 0, c.ktot, P.k, P.a_ks, 0};
          if (two) x.s1 = (int32_t)(rw[u].one ? rw[u].s0 * d0 : rw[u].s1);
          if (P.a_ks != NO_STRIDE) {
            nr_a.push_back(x);
          } else {  // k modes that do not merge: one entry per k
            x.k = 1;
            x.ks = 0;
            for (int k = 0; k < P.k; ++k, ++x.k0) {
              x.off = P.a_off;
              int rem = k;
              for (int d = 0; d < q.n_k; ++d) {
                x.off += (int64_t)(rem % q.k_dims[d]) * q.a_k_stride[d];
                rem /= q.k_dims[d];
              }
              nr_a.push_back(x);
            }
          }
          c.ktot += P.k;
        }
        c.a_end = (int32_t)nr_a.size();
        cost += (int64_t)c.m * (c.ktot + c.cols);
        ids.push_back((int)nr_chunks.size());
        nr_chunks.push_back(c);
        x = y;
      }
      groups.emplace_back(cost, std::move(ids));
    }
    std::stable_sort(groups.begin(), groups.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
    // rows per CTA: enough tiles to pay for staging B, but eight CTAs per SM and
    // more while there are rows (at bond dimension 1400 2857 us per two products
    // with this bound, 2894 with sixteen tiles as soon as there are four CTAs)
    int64_t all = 0;
    for (const NrChunk& c : nr_chunks) all += (c.m + 127) / 128;
    // (a thread per row: its tiles are blocks of their own, so that is how many a task
    // describes; one each, they were 24000 for an environment update at 2048, which took
    // 1 ms longer to plan)
    const int rows = rd_threads > 0 ? rd_threads : nr_rw * NR_WARPS;
    const int tiles = (int)std::max<int64_t>(1, std::min<int64_t>(16, all / (8 * (int64_t)ctx->num_sms)));
    if (rd_threads > 0) rd_tiles = tiles;
    for (const auto& gr : groups) {
      const int m = nr_chunks[gr.second[0]].m;
      for (int row0 = 0; row0 < m; row0 += tiles * rows)
        for (int id : gr.second)
          nr_tasks.push_back(NrTask{nr_chunks[id], row0, std::min(tiles, (m - row0 + rows - 1) / rows), 0});
    }
  }
  // the offset tables that this path reads, back to back (elsewhere strides serve)
  {
    auto need = [&](int32_t& id, bool used) {
      if (!used) {
        id = 0;
        return;
      }
      TableJob& J = jobs[id];
      if (J.dst < 0) {
        J.dst = (int32_t)tab_len;
        tab_len += J.len;
      }
      id = J.dst;
    };
    for (const NrChunk& c : nr_chunks)
      if (c.d0 == 0)
        for (int i = c.a_begin; i < c.a_end; ++i) need(nr_a[i].s0, true);
    for (NrB& x : nr_b) {
      need(x.ktab, x.ks == NO_STRIDE);
      need(x.ctab, x.cs == NO_STRIDE);
    }
    for (PairDev& P : hp) {
      need(P.rowA, tc || (!narrow && P.a_rs == NO_STRIDE));
      need(P.colA, tc || (!narrow && P.a_ks == NO_STRIDE));
      need(P.rowB, tc || (!narrow && P.b_ks == NO_STRIDE));
      need(P.colB, tc || (!narrow && P.b_cs == NO_STRIDE));
      TT_REQUIRE(tab_len < (1ll << 31), "tt_contract_plan: offset tables too large");
    }
    jobs.erase(std::remove_if(jobs.begin(), jobs.end(), [](const TableJob& J) { return J.dst < 0; }), jobs.end());
  }
  const bool dgemm = !tc && !narrow;
  std::vector<DTask> dtasks;
  int split = 1;
  if (dgemm) {
    int longest = 0;
    for (const TaskDev& t : tsorted) {
      const tt_out_block& o = outs[t.out];
      dtasks.push_back(DTask{o.c_off, o.m, o.n, o.ldc, t.m0, t.n0, t.p_begin, t.p_end, chunks[t.out]});
      longest = std::max(longest, chunks[t.out]);
    }
    split = dgemm_split((int64_t)dtasks.size(), longest, ctx->num_sms);
  }
  std::vector<OutDev> ho(n_out);
  for (int o = 0; o < n_out; ++o) ho[o] = OutDev{outs[o].c_off, outs[o].m, outs[o].n, outs[o].ldc};

  lap(2);
  // tensor-core path: one packing job per distinct operand block
  std::vector<PackJob> ja, jb;
  std::vector<PackTile> ta, tb;
  std::vector<PairTC> ptc;
  int64_t bytesA = 0, bytesB = 0;
  if (tc) {
    std::map<int64_t, int> ua, ub;
    ptc.resize(n_pairs);
    for (int ii = 0; ii < n_pairs; ++ii) {
      const PairDev& P = hp[ii];
      const int kt = (P.k + TC_BK - 1) / TC_BK;
      auto ia = ua.find(P.a_off);
      if (ia == ua.end()) {
        const int rt = (P.m + TC_BM - 1) / TC_BM;
        ja.push_back(PackJob{P.a_off, bytesA, P.m, P.k, P.rowA, P.colA, kt, P.a_mfast});
        for (int r = 0; r < rt; ++r)
          for (int k = 0; k < kt; ++k) ta.push_back(PackTile{(int32_t)ja.size() - 1, r, k});
        bytesA += (int64_t)rt * kt * TC_TILE_BYTES;
        ia = ua.emplace(P.a_off, (int)ja.size() - 1).first;
      }
      auto ib = ub.find(P.b_off);
      if (ib == ub.end()) {
        const int rt = (P.n + TC_BN - 1) / TC_BN;
        jb.push_back(PackJob{P.b_off, bytesB, P.n, P.k, P.colB, P.rowB, kt, P.b_kfast ? 0 : 1});
        for (int r = 0; r < rt; ++r)
          for (int k = 0; k < kt; ++k) tb.push_back(PackTile{(int32_t)jb.size() - 1, r, k});
        bytesB += (int64_t)rt * kt * TC_TILE_BYTES;
        ib = ub.emplace(P.b_off, (int)jb.size() - 1).first;
      }
      ptc[ii] = PairTC{ja[ia->second].dst, jb[ib->second].dst, kt, 0};
    }
    TT_REQUIRE(ta.size() < (1u << 31) && tb.size() < (1u << 31), "tt_contract_plan: too many packed tiles");
  }

  tt_plan* plan = new tt_plan();
  plan->precision = precision;
  plan->narrow = narrow;
  plan->nr_rw = nr_rw;
  plan->nr_cols = nr_cols;
  plan->rd_threads = rd_threads;
  plan->rd_tiles = rd_tiles;
  for (const NrChunk& c : nr_chunks) plan->nr_ktot = std::max(plan->nr_ktot, c.ktot);
  plan->n_tilesA = (int)ta.size();
  plan->n_tilesB = (int)tb.size();
  plan->bytesA = bytesA;
  plan->bytesB = bytesB;
  plan->n_tasks = narrow ? (int)nr_tasks.size() : (int)tsorted.size();
  plan->split = split;
  plan->n_pairs = n_pairs;
  plan->n_out = n_out;
  plan->flops = flops;
  // the plan's arrays in one device buffer, filled by one staged copy (the host
  // vectors may die at return without stalling the stream); the offset tables
  // and the status word, where the path has them, follow it
  std::vector<char> blob;
  auto put = [&](const auto& v) {
    const size_t at = blob.size();
    blob.resize((at + v.size() * sizeof(v[0]) + 15) & ~(size_t)15);
    if (!v.empty()) memcpy(blob.data() + at, v.data(), v.size() * sizeof(v[0]));
    return at;
  };
  size_t at_tasks = 0, at_outs = 0, at_pairs = 0, at_a = 0, at_b = 0, at_c = 0, at_ja = 0, at_jb = 0, at_ta = 0, at_tb = 0,
         at_ptc = 0;
  if (dgemm) {
    at_tasks = put(dtasks);
    at_pairs = put(hp);
  } else if (narrow) {
    at_tasks = put(nr_tasks);
    at_a = put(nr_a);
    at_b = put(nr_b);
    at_c = put(nr_c);
  } else {
    at_tasks = put(tsorted);
    at_outs = put(ho);
    at_ja = put(ja);
    at_jb = put(jb);
    at_ta = put(ta);
    at_tb = put(tb);
    at_ptc = put(ptc);
  }
  const size_t at_jobs = put(jobs);
  const size_t at_status = blob.size(), at_tab = at_status + 16;
  const size_t total = at_tab + sizeof(int32_t) * (size_t)tab_len;
  plan->dev_bytes = (int64_t)total;
  plan->d_blob = tt::pool_alloc<char>(ctx, total);
  if (!plan->d_blob) {
    tt_plan_destroy(ctx, plan);
    return tt::fail(TT_ERR_OOM, "tt_contract_plan: device allocation failed");
  }
  blob.resize(at_tab, 0);  // the status word starts as TT_OK
  char* d = plan->d_blob;
  if (dgemm) plan->d_dtasks = reinterpret_cast<DTask*>(d + at_tasks);
  else if (narrow) plan->d_nr_tasks = reinterpret_cast<NrTask*>(d + at_tasks);
  else plan->d_tasks = reinterpret_cast<TaskDev*>(d + at_tasks);
  plan->d_outs = reinterpret_cast<OutDev*>(d + at_outs);
  plan->d_pairs = reinterpret_cast<PairDev*>(d + at_pairs);
  plan->d_nr_a = reinterpret_cast<NrA*>(d + at_a);
  plan->d_nr_b = reinterpret_cast<NrB*>(d + at_b);
  plan->d_nr_c = reinterpret_cast<int64_t*>(d + at_c);
  plan->d_jobsA = reinterpret_cast<PackJob*>(d + at_ja);
  plan->d_jobsB = reinterpret_cast<PackJob*>(d + at_jb);
  plan->d_tilesA = reinterpret_cast<PackTile*>(d + at_ta);
  plan->d_tilesB = reinterpret_cast<PackTile*>(d + at_tb);
  plan->d_pairtc = reinterpret_cast<PairTC*>(d + at_ptc);
  plan->d_status = reinterpret_cast<int*>(d + at_status);
  plan->d_tab = reinterpret_cast<int32_t*>(d + at_tab);
  cudaStream_t s = ctx->stream;
  lap(3);
  TT_CUDA(tt::h2d_async(ctx, d, blob.data(), blob.size()));
  if (!jobs.empty()) {
    expand_tables<<<(unsigned)jobs.size(), 128, 0, s>>>(reinterpret_cast<const TableJob*>(d + at_jobs), (int)jobs.size(),
                                                        plan->d_tab);
    TT_LAUNCH_CHECK(ctx);
  }
  *plan_out = plan;
  return TT_OK;
}

int tt_contract_exec(tt_ctx* ctx, const tt_plan* plan, const double* A, const double* B,
                     double* C, double alpha) {
  return tt_contract_exec_keep(ctx, plan, A, B, C, alpha, 0);
}

int tt_plan_release_packed(tt_ctx* ctx, const tt_plan* plan) {
  TT_REQUIRE(ctx && plan, "tt_plan_release_packed: null argument");
  for (int w = 0; w < 2; ++w) {
    tt::pool_free(ctx, plan->kept[w]);
    plan->kept[w] = nullptr;
    plan->kept_src[w] = nullptr;
    tt::pool_free(ctx, plan->scratch[w]);
    plan->scratch[w] = nullptr;
  }
  return TT_OK;
}

int tt_contract_exec_keep(tt_ctx* ctx, const tt_plan* plan, const double* A, const double* B, double* C,
                          double alpha, int keep) {
  return tt_contract_exec_stamped(ctx, plan, A, B, C, alpha, keep, nullptr);
}

int tt_plan_stamps(const tt_plan* plan) {
  return plan && plan->n_tasks > 0 && plan->precision == TT_PREC_FP64 ? 1 : 0;
}

int tt_contract_exec_stamped(tt_ctx* ctx, const tt_plan* plan, const double* A, const double* B, double* C,
                             double alpha, int keep, uint64_t* d_stamp) {
  TT_REQUIRE(ctx && plan, "tt_contract_exec: null argument");
  TT_REQUIRE(!d_stamp || tt_plan_stamps(plan), "tt_contract_exec_stamped: not an FP64 plan");
  if (plan->n_tasks == 0) return TT_OK;
  static thread_local uint64_t attr_set = 0;  // per host thread and device
  if (tt::first_on_device(attr_set, ctx->device)) {
    TT_CUDA(cudaFuncSetAttribute(grouped_dgemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SMEM_BYTES));
    TT_CUDA(cudaFuncSetAttribute(narrow_dgemm<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)narrow_smem(NR_KTOT, 8, narrow_ld(NR_N))));
    TT_CUDA(cudaFuncSetAttribute(narrow_dgemm<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)narrow_smem(NR_KTOT, 32, narrow_ld(NR_N))));
    TT_CUDA(cudaFuncSetAttribute(grouped_tc_persist<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TC_BULK_SMEM));
    TT_CUDA(cudaFuncSetAttribute(grouped_tc_persist<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TC_BULK_SMEM));
  }
  if (plan->precision == TT_PREC_FP64) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)plan->split;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.stream = ctx->stream;
    cfg.attrs = at;
    cfg.numAttrs = !plan->narrow && plan->split > 1 ? 2 : 1;
    if (plan->narrow && plan->rd_threads > 0) {
      const int nc = plan->nr_cols <= 4 ? 4 : plan->nr_cols <= 8 ? 8 : RD_COLS;
      // segments of equal length
      const int kmax = RD_SEG / (8 * nc), segs = std::max(1, (plan->nr_ktot + kmax - 1) / kmax);
      const int kseg = std::max(1, (plan->nr_ktot + segs - 1) / segs);
      cfg.gridDim = dim3((unsigned)plan->n_tasks, (unsigned)plan->rd_tiles);
      cfg.blockDim = dim3((unsigned)plan->rd_threads);
      cfg.dynamicSmemBytes = sizeof(double) * (size_t)kseg * nc;
      const auto fn = plan->rd_threads == 128
                          ? (nc == 4   ? rows_dgemm<4, false>
                             : nc == 8 ? rows_dgemm<8, false>
                                       : rows_dgemm<RD_COLS, false>)
                          : (nc == 4   ? rows_dgemm<4, true>
                             : nc == 8 ? rows_dgemm<8, true>
                                       : rows_dgemm<RD_COLS, true>);
      static thread_local uint64_t rd_set[3] = {0, 0, 0};  // as attr_set, per instance that may need it
      if (plan->rd_threads != 128 && tt::first_on_device(rd_set[nc == 4 ? 0 : nc == 8 ? 1 : 2], ctx->device))
        TT_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, RD_SEG));
      TT_CUDA(cudaLaunchKernelEx(&cfg, fn,
                                 (const NrTask*)plan->d_nr_tasks, (const NrA*)plan->d_nr_a, (const NrB*)plan->d_nr_b,
                                 (const int64_t*)plan->d_nr_c, (const int32_t*)plan->d_tab, A, B, C, alpha, kseg,
                                 (unsigned long long*)d_stamp));
    } else if (plan->narrow) {
      cfg.gridDim = dim3((unsigned)plan->n_tasks);
      cfg.blockDim = dim3(NR_THREADS);
      cfg.dynamicSmemBytes = narrow_smem(plan->nr_ktot, plan->nr_rw, narrow_ld(plan->nr_cols));
      TT_CUDA(cudaLaunchKernelEx(&cfg, plan->nr_rw == 8 ? narrow_dgemm<8> : narrow_dgemm<32>,
                                 (const NrTask*)plan->d_nr_tasks, (const NrA*)plan->d_nr_a, (const NrB*)plan->d_nr_b,
                                 (const int64_t*)plan->d_nr_c, (const int32_t*)plan->d_tab, A, B, C, alpha,
                                 narrow_buf(plan->nr_ktot, plan->nr_rw), narrow_ld(plan->nr_cols), (unsigned long long*)d_stamp));
    } else {
      cfg.gridDim = dim3((unsigned)plan->n_tasks * (unsigned)plan->split);
      cfg.blockDim = dim3(THREADS);
      cfg.dynamicSmemBytes = SMEM_BYTES;
      TT_CUDA(cudaLaunchKernelEx(&cfg, grouped_dgemm, (const DTask*)plan->d_dtasks,
                                 (const PairDev*)plan->d_pairs, (const int32_t*)plan->d_tab, A, B, C, alpha,
                                 plan->split, (unsigned long long*)d_stamp));
    }
    TT_LAUNCH_CHECK(ctx);
    return TT_OK;
  }
  // pack the operands into tensor-core tiles (pool buffers, released in
  // stream order); an operand kept from an earlier exec of this plan, packed
  // from the same source, is reused as it is
  const bool split = plan->precision == TT_PREC_TF32X3;
  const double* src[2] = {A, B};
  const int64_t bytes[2] = {plan->bytesA, plan->bytesB};
  uint8_t* pk[2] = {nullptr, nullptr};
  bool fresh[2] = {false, false};
  bool from_scratch[2] = {false, false};
  for (int w = 0; w < 2; ++w) {
    const bool k = (keep >> w) & 1;
    if (k && plan->kept[w] && plan->kept_src[w] == src[w]) {
      pk[w] = plan->kept[w];
      continue;
    }
    if (k && plan->kept[w]) {  // kept from another source: stale
      tt::pool_free(ctx, plan->kept[w]);
      plan->kept[w] = nullptr;
      plan->kept_src[w] = nullptr;
    }
    fresh[w] = true;
    if (!k && ((keep >> (2 + w)) & 1)) {  // repacked every exec into a buffer the plan keeps
      if (!plan->scratch[w]) plan->scratch[w] = tt::pool_alloc<uint8_t>(ctx, (size_t)std::max<int64_t>(bytes[w], 16));
      pk[w] = plan->scratch[w];
      from_scratch[w] = true;
      continue;
    }
    pk[w] = tt::pool_alloc<uint8_t>(ctx, (size_t)std::max<int64_t>(bytes[w], 16));
  }
  uint8_t* pa = pk[0];
  uint8_t* pb = pk[1];
  if (!pa || !pb) {
    if (fresh[0] && !from_scratch[0]) tt::pool_free(ctx, pa);
    if (fresh[1] && !from_scratch[1]) tt::pool_free(ctx, pb);
    return tt::fail(TT_ERR_OOM, "tt_contract_exec: packed operand allocation failed");
  }
  {
    // one launch for the operands that need packing: tiles [0, na) of A, then those of B
    const int na = fresh[0] ? plan->n_tilesA : 0, nb = fresh[1] ? plan->n_tilesB : 0;
    if (na + nb > 0) {
      const unsigned nt = (unsigned)(na + nb);
      if (split)
        pack_tf32_ab<true><<<nt, 128, 0, ctx->stream>>>(plan->d_jobsA, plan->d_tilesA, na, plan->d_jobsB,
                                                         plan->d_tilesB, plan->d_tab, A, B, pa, pb);
      else
        pack_tf32_ab<false><<<nt, 128, 0, ctx->stream>>>(plan->d_jobsA, plan->d_tilesA, na, plan->d_jobsB,
                                                          plan->d_tilesB, plan->d_tab, A, B, pa, pb);
      TT_LAUNCH_CHECK(ctx);
    }
  }
  const unsigned grid = (unsigned)std::min(plan->n_tasks, std::max(1, ctx->num_sms));
  if (split)
    grouped_tc_persist<true><<<grid, TC_P_THREADS, TC_BULK_SMEM, ctx->stream>>>(
        plan->d_tasks, plan->n_tasks, plan->d_outs, plan->d_pairtc, pa, pb, C, alpha, plan->d_status,
        ctx->d_dev_status, ctx->wait_limit);
  else
    grouped_tc_persist<false><<<grid, TC_P_THREADS, TC_BULK_SMEM, ctx->stream>>>(
        plan->d_tasks, plan->n_tasks, plan->d_outs, plan->d_pairtc, pa, pb, C, alpha, plan->d_status,
        ctx->d_dev_status, ctx->wait_limit);
  cudaError_t le = cudaGetLastError();
  for (int w = 0; w < 2; ++w) {
    if (!fresh[w] || from_scratch[w]) continue;
    if ((keep >> w) & 1) {
      plan->kept[w] = pk[w];
      plan->kept_src[w] = src[w];
    } else {
      tt::pool_free(ctx, pk[w]);
    }
  }
  if (le != cudaSuccess) return tt::cuda_fail(le, "tt_contract_exec: tensor-core launch", __FILE__, __LINE__);
  tt::count_launch(ctx);
  return TT_OK;
}

int tt_plan_destroy(tt_ctx* ctx, tt_plan* plan) {
  if (!plan) return TT_OK;
  if (ctx) {
    tt_plan_release_packed(ctx, plan);
    tt::pool_free(ctx, plan->d_blob);
  }
  delete plan;
  return TT_OK;
}

int tt_plan_device_status(tt_ctx* ctx, const tt_plan* plan, int* status) {
  TT_REQUIRE(ctx && plan && status, "tt_plan_device_status: null argument");
  int h = 0;
  TT_CUDA(cudaMemcpyAsync(&h, plan->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  TT_CUDA(cudaStreamSynchronize(ctx->stream));
  *status = h;
  return TT_OK;
}

int tt_contract_predict(const tt_out_block* outs, int n_out, const tt_block_pair* pairs, int n_pairs,
                        int precision, int num_sms, double* us_fp64, double* us_tc, int* choice) {
  TT_REQUIRE(outs && (n_pairs == 0 || pairs) && us_fp64 && us_tc && choice, "tt_contract_predict: null argument");
  TT_REQUIRE(n_out >= 0 && n_pairs >= 0 && num_sms >= 1, "tt_contract_predict: bad counts");
  TT_REQUIRE(precision == TT_PREC_TF32_AUTO || precision == TT_PREC_TF32X3_AUTO,
             "tt_contract_predict: precision must be TT_PREC_TF32_AUTO or TT_PREC_TF32X3_AUTO");
  const int kind = precision == TT_PREC_TF32_AUTO ? TT_PREC_TF32 : TT_PREC_TF32X3;
  // the pairs grouped by output block, as tt_contract_plan groups them
  std::vector<int> order(n_pairs);
  std::iota(order.begin(), order.end(), 0);
  for (int i = 0; i < n_pairs; ++i)
    TT_REQUIRE(pairs[i].out_block >= 0 && pairs[i].out_block < n_out,
               "tt_contract_predict: pair references a missing output block");
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return pairs[a].out_block < pairs[b].out_block; });
  std::vector<PairDev> hp(n_pairs);
  std::vector<int> first(n_out + 1, 0);
  for (int ii = 0; ii < n_pairs; ++ii) {
    const tt_block_pair& q = pairs[order[ii]];
    TT_REQUIRE(q.n_m >= 0 && q.n_m <= TT_MAX_MODES && q.n_k >= 0 && q.n_k <= TT_MAX_MODES && q.n_n >= 0 &&
                   q.n_n <= TT_MAX_MODES,
               "tt_contract_predict: mode count out of range");
    int64_t m = 1, n = 1, k = 1;
    for (int i = 0; i < q.n_m; ++i) m *= q.m_dims[i];
    for (int i = 0; i < q.n_k; ++i) k *= q.k_dims[i];
    for (int i = 0; i < q.n_n; ++i) n *= q.n_dims[i];
    PairDev P;
    memset(&P, 0, sizeof(P));
    P.a_off = q.a_off;
    P.b_off = q.b_off;
    P.m = (int)m;
    P.n = (int)n;
    P.k = (int)k;
    hp[ii] = P;
    first[q.out_block + 1]++;
  }
  for (int o = 0; o < n_out; ++o) first[o + 1] += first[o];
  *us_fp64 = predict_us(outs, n_out, hp, first, TT_PREC_FP64, num_sms);
  *us_tc = predict_us(outs, n_out, hp, first, kind, num_sms);
  *choice = *us_tc > 0.8 * *us_fp64 ? TT_PREC_FP64 : kind;  // the rule tt_contract_plan applies
  return TT_OK;
}

int tt_plan_precision(const tt_plan* plan, int* precision) {
  TT_REQUIRE(plan && precision, "tt_plan_precision: null argument");
  *precision = plan->precision;
  return TT_OK;
}

int tt_contract_plan_timers(double* seconds, int n) {
  TT_REQUIRE(seconds && n >= 0, "tt_contract_plan_timers: null argument");
  for (int i = 0; i < n && i < 5; ++i) seconds[i] = g_plan_stage_s[i];
  return TT_OK;
}

int tt_plan_device_bytes(const tt_plan* plan, int64_t* bytes) {
  TT_REQUIRE(plan && bytes, "tt_plan_device_bytes: null argument");
  *bytes = plan->dev_bytes;
  return TT_OK;
}

int tt_plan_flops(const tt_plan* plan, double* flops) {
  TT_REQUIRE(plan && flops, "tt_plan_flops: null argument");
  *flops = plan->flops;
  return TT_OK;
}

}  // extern "C"
