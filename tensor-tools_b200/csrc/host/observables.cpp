// Overlaps, MPO expectation values and Sz correlators (qMPS and dense MPS).
#include "observables.h"

#include <algorithm>
#include <stdexcept>

namespace ttb {

namespace {

tt_ctx* bound_ctx() {
  if (!rt().ctx) throw std::runtime_error("observables: no device context bound");
  return rt().ctx;
}

// psi_i^dagger with its link indices primed (t1 of mps/observables.cpp:386,419)
qtensor bra_tensor(const qtensor& A) {
  qtensor t = A;
  t.dag();
  for (auto& ix : t.idx_set)
    if (ix.type() == Link) ix.prime();
  return t;
}

// ones over (a, b), daggered: the closing tensors of observables.cpp:423-428,432-437
qtensor ends(const qtensor_index& a, const qtensor_index& b) {
  qtensor e({a, b});
  e.initBlock();
  e.setOne();
  e.dag();
  return e;
}

int site_axis(const qtensor& A) {
  for (unsigned k = 0; k < A.rank; ++k)
    if (A.idx_set[k].type() == Site) return (int)k;
  throw std::runtime_error("measure_sz: MPS tensor without a site index");
}

// Sz applied to the physical mode: every block carries one spin sector of
// dimension 1, so Sz is a constant factor (2Sz / 2) per block.
qtensor apply_sz(const qtensor& A) {
  qtensor t = A;
  int s = site_axis(A);
  for (unsigned b = 0; b < t.blocks.size(); ++b) {
    const BlockMeta& bm = t.blocks[b];
    if (bm.qd[s] != 1) throw std::runtime_error("measure_sz: spin-1/2 sites expected");
    double f = 0.5 * (double)bm.qn[s].a;
    check(tt_vec_scale_mode(bound_ctx(), bm.size, 1, 1, &f, t.block_ptr(b)), "apply Sz");
  }
  return t;
}

void check_pair(unsigned La, unsigned Lb) {
  if (La != Lb || La < 2) throw std::runtime_error("observables: length mismatch");
}

}  // namespace

double psiphi(const qMPS& psi, const qMPS& phi) {
  // mps/observables.cpp:415-450
  check_pair(psi.length, phi.length);
  qtensor acc;
  double res = 0.0;
  for (unsigned i = 0; i < psi.length; ++i) {
    qtensor t1 = bra_tensor(psi.A[i]);
    const qtensor& t2 = phi.A[i];
    if (i == 0) {
      acc = (ends(t1.idx_set[0], t2.idx_set[0]) * t1) * t2;
    } else {
      acc = (t1 * acc) * t2;
    }
    if (i == psi.length - 1) res = acc.contract(ends(t1.idx_set.back(), t2.idx_set.back()));
  }
  return res;
}

double psiHphi(const qMPS& psi, const qMPO& H, const qMPS& phi) {
  // mps/observables.cpp:64-103
  check_pair(psi.length, phi.length);
  check_pair(psi.length, H.length);
  qtensor acc;
  double res = 0.0;
  for (unsigned i = 0; i < psi.length; ++i) {
    qtensor t1 = psi.A[i];
    t1.dag();
    t1.prime();
    const qtensor& t2 = H.A[i];
    const qtensor& t3 = phi.A[i];
    if (i == 0) {
      qtensor le({t1.idx_set[0], t2.idx_set[0], t3.idx_set[0]});
      le.initBlock();
      le.setOne();
      le.dag();
      acc = ((le * t1) * t2) * t3;
    } else {
      acc = ((acc * t1) * t2) * t3;
    }
    if (i == psi.length - 1) {
      qtensor re({t1.idx_set.back(), t2.idx_set.back(), t3.idx_set.back()});
      re.initBlock();
      re.setOne();
      re.dag();
      res = acc.contract(re);
    }
  }
  return res;
}

namespace {

// The left environments at one bond of several insertions of Sz, as one tensor
// with an index of charge 0 that counts them: the identity first, then the sites.
constexpr const char* kOrigin = "SzOrigin";

qtensor_index origin_index(unsigned n) {
  qtensor_index ix(Inward, kOrigin, Link);
  ix.addQN(QN(0, 0), n);
  return ix;
}

// t's blocks for n environments in all: the same blocks with the origin index
// second, where the products with a site's tensors put it
qtensor origin_blocks(const qtensor& t, unsigned n) {
  const bool has = t.rank == 3;
  qtensor r(std::vector<qtensor_index>{t.idx_set[0], origin_index(n), t.idx_set[has ? 2 : 1]});
  for (const BlockMeta& b : t.blocks) {
    const int last = has ? 2 : 1;
    r.add_block_meta({b.qn[0], QN(0, 0), b.qn[last]}, {b.qi[0], 0u, b.qi[last]}, {b.qd[0], (int)n, b.qd[last]});
  }
  r.allocate(false);
  r._initted = true;
  return r;
}

// S's environments (m of them) and behind them the one of C
qtensor with_origin(const qtensor& S, const qtensor& C) {
  const unsigned m = S.rank == 3 ? S.idx_set[1].qdim(0) : 0;
  qtensor r = origin_blocks(m > 0 ? S : C, m + 1);
  for (const BlockMeta& b : C.blocks)
    if (m > 0 && r.find_block({b.qn[0].pack(), QN(0, 0).pack(), b.qn[1].pack()}) < 0)
      throw std::runtime_error("measure_sz: an environment's block is missing");
  auto put = [&](const qtensor& t, unsigned first, unsigned n) {
    std::vector<tt_copy_desc> descs;
    for (const BlockMeta& b : t.blocks) {
      const int last = (int)t.rank - 1;
      const BlockMeta& rb = r.blocks[r.find_block({b.qn[0].pack(), QN(0, 0).pack(), b.qn[last].pack()})];
      tt_copy_desc d = {};
      d.n_modes = 2;  // n columns of one environment each are contiguous
      d.dims[0] = b.qd[0] * (int)n;
      d.dims[1] = b.qd[last];
      d.src_off = b.off;
      d.src_stride[0] = d.dst_stride[0] = 1;
      d.src_stride[1] = (int64_t)b.qd[0] * n;
      d.dst_off = rb.off + (int64_t)b.qd[0] * first;
      d.dst_stride[1] = (int64_t)b.qd[0] * (m + 1);
      descs.push_back(d);
    }
    for (size_t i = 0; i < descs.size(); i += 65535)
      check(tt_strided_copy_batched(bound_ctx(), descs.data() + i, (int)std::min<size_t>(65535, descs.size() - i),
                                    t.data->get(), r.data->get()),
            "environment copy");
  };
  if (C.blocks.size() < r.blocks.size()) r.data->zero();
  if (m > 0) put(S, 0, m);
  put(C, m, 1);
  return r;
}

}  // namespace

// <Sz_i> and <Sz_i Sz_j>.  The environments of all sites i left of a bond go
// through a site together, in two products, and meet the right environment with
// Sz at j in a third, so a chain takes about 8 L launches and one read of the
// results, where one by one they were 4 L^2 / 2 launches and L^2 / 2 reads.
void measure_sz(const qMPS& psi, std::vector<double>& sz, std::vector<double>& szsz) {
  const unsigned L = psi.length;
  if (L < 2) throw std::runtime_error("measure_sz: need at least two sites");
  std::vector<qtensor> bra(L), zket(L);
  for (unsigned i = 0; i < L; ++i) {
    bra[i] = bra_tensor(psi.A[i]);
    zket[i] = apply_sz(psi.A[i]);
  }
  // EL[i]: sites < i contracted (bond i); ZR[j]: sites >= j contracted, with Sz at j
  std::vector<qtensor> EL(L + 1), ZR(L);
  EL[0] = ends(bra[0].idx_set[0], psi.A[0].idx_set[0]);
  int64_t largest = 1;
  for (unsigned i = 0; i < L; ++i) {
    EL[i + 1] = (bra[i] * EL[i]) * psi.A[i];
    largest = std::max(largest, EL[i + 1].arena);
  }
  qtensor ER = ends(bra[L - 1].idx_set.back(), psi.A[L - 1].idx_set.back());
  double nrm2 = EL[L].contract(ER);
  if (!(nrm2 > 0.0)) throw std::runtime_error("measure_sz: <psi|psi> is not positive");
  for (unsigned i = L; i-- > 0;) {
    qtensor D = bra[i] * ER;
    ZR[i] = D * zket[i];
    if (i > 0) ER = D * psi.A[i];
  }
  // 64 sites at a time (100 sites, bond dimension 40: 16 sites 35 ms, 64 25, all 24; 160
  // sites at 20: 55, 34, 29), fewer where that would be more than 2^26 numbers, 0.5 GB in
  // each of the four stacks that are alive at once, or more than the device has room for
  unsigned chunk =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>(std::min(L, 64u), ((int64_t)1 << 26) / largest));
  const unsigned row = chunk + 1;
  sz.assign(L, 0.0);
  szsz.assign((size_t)L * L, 0.0);
  DevBuf vals((int64_t)L * row);
  std::vector<double> h((size_t)L * row);
  auto group = [&](unsigned i0, unsigned i1) {  // the sites i0 <= i < i1
    vals.zero();
    qtensor S = with_origin(qtensor(), EL[i0]);
    for (unsigned j = i0; j < L; ++j) {
      auto cc = contract_cached(S, ZR[j], false);
      if (tt_plan* p = cc->plan_for(TT_PREC_FP64))  // an inner product, whatever operator* runs in
        check(tt_contract_exec(bound_ctx(), p, S.data->get(), ZR[j].data->get(), vals.get() + (size_t)j * row, 1.0),
              "contract exec");
      if (j + 1 == L) break;
      S = (bra[j] * S) * psi.A[j];
      if (j < i1) S = with_origin(S, (bra[j] * EL[j]) * zket[j]);
    }
    check(tt_memcpy_d2h(bound_ctx(), h.data(), vals.get(), sizeof(double) * h.size()), "d2h");
    for (unsigned j = i0; j < L; ++j) {
      if (j < i1) {
        sz[j] = h[(size_t)j * row] / nrm2;
        szsz[(size_t)j * L + j] = 0.25;
      }
      for (unsigned i = i0; i < std::min(i1, j); ++i)
        szsz[(size_t)i * L + j] = szsz[(size_t)j * L + i] = h[(size_t)j * row + 1 + i - i0] / nrm2;
    }
  };
  for (unsigned i0 = 0; i0 < L;) {
    const unsigned i1 = std::min(L, i0 + chunk);
    try {
      group(i0, i1);
      i0 = i1;
    } catch (const tt_error& e) {
      if (e.code != TT_ERR_OOM || chunk == 1) throw;
      chunk = (chunk + 1) / 2;
    }
  }
}

// ---- dense MPS ------------------------------------------------------------------
namespace {

tt_ctx* dense_ctx() {
  if (!rt().ctx) throw std::runtime_error("observables: no device context bound");
  return rt().ctx;
}

dtensor dbra(const dtensor& A) {
  dtensor t = A;
  for (auto& ix : t.idx_set)
    if (ix.type == Link) ix.prime();
  return t;
}

dtensor dends(const dtensor_index& a, const dtensor_index& b) {
  dtensor e({a, b});
  e.setOne();
  return e;
}

dtensor dapply_sz(const dtensor& A) {
  dtensor t = A;
  int s = -1;
  for (unsigned k = 0; k < t.rank; ++k)
    if (t.idx_set[k].type == Site) s = (int)k;
  if (s < 0 || t.idx_set[s].size != 2) throw std::runtime_error("measure_sz: spin-1/2 site index expected");
  int64_t inner = 1, outer = 1;
  for (int k = 0; k < s; ++k) inner *= t.idx_set[k].size;
  for (unsigned k = s + 1; k < t.rank; ++k) outer *= t.idx_set[k].size;
  const double f[2] = {-0.5, 0.5};  // Dn, Up
  check(tt_vec_scale_mode(dense_ctx(), inner, 2, outer, f, t.data->get()), "apply Sz");
  return t;
}

}  // namespace

double psiphi(const MPS& psi, const MPS& phi) {
  // mps/observables.cpp:382-413
  check_pair(psi.length, phi.length);
  dtensor acc;
  double res = 0.0;
  for (unsigned i = 0; i < psi.length; ++i) {
    dtensor t1 = dbra(psi.A[i]);
    const dtensor& t2 = phi.A[i];
    if (i == 0)
      acc = (dends(t1.idx_set[0], t2.idx_set[0]) * t1) * t2;
    else
      acc = (t1 * acc) * t2;
    if (i == psi.length - 1) res = acc.inner_product(dends(t1.idx_set.back(), t2.idx_set.back()));
  }
  return res;
}

double psiHphi(const MPS& psi, const MPO& H, const MPS& phi) {
  // mps/observables.cpp:25-62
  check_pair(psi.length, phi.length);
  check_pair(psi.length, H.length);
  dtensor acc;
  double res = 0.0;
  for (unsigned i = 0; i < psi.length; ++i) {
    dtensor t1 = psi.A[i];
    t1.prime();
    const dtensor& t2 = H.A[i];
    const dtensor& t3 = phi.A[i];
    if (i == 0) {
      dtensor le({t1.idx_set[0], t2.idx_set[0], t3.idx_set[0]});
      le.setOne();
      acc = ((le * t1) * t2) * t3;
    } else {
      acc = ((acc * t1) * t2) * t3;
    }
    if (i == psi.length - 1) {
      dtensor re({t1.idx_set.back(), t2.idx_set.back(), t3.idx_set.back()});
      re.setOne();
      res = acc.inner_product(re);
    }
  }
  return res;
}

void measure_sz(const MPS& psi, std::vector<double>& sz, std::vector<double>& szsz) {
  const unsigned L = psi.length;
  if (L < 2) throw std::runtime_error("measure_sz: need at least two sites");
  std::vector<dtensor> bra(L), zket(L);
  for (unsigned i = 0; i < L; ++i) {
    bra[i] = dbra(psi.A[i]);
    zket[i] = dapply_sz(psi.A[i]);
  }
  std::vector<dtensor> EL(L + 1), ER(L + 1);
  EL[0] = dends(bra[0].idx_set[0], psi.A[0].idx_set[0]);
  for (unsigned i = 0; i < L; ++i) EL[i + 1] = (bra[i] * EL[i]) * psi.A[i];
  ER[L] = dends(bra[L - 1].idx_set.back(), psi.A[L - 1].idx_set.back());
  for (unsigned i = L; i-- > 0;) ER[i] = (bra[i] * ER[i + 1]) * psi.A[i];
  double nrm2 = EL[L].inner_product(ER[L]);
  if (!(nrm2 > 0.0)) throw std::runtime_error("measure_sz: <psi|psi> is not positive");
  sz.assign(L, 0.0);
  szsz.assign((size_t)L * L, 0.0);
  for (unsigned i = 0; i < L; ++i) {
    dtensor C = (bra[i] * EL[i]) * zket[i];
    sz[i] = C.inner_product(ER[i + 1]) / nrm2;
    szsz[(size_t)i * L + i] = 0.25;
    for (unsigned j = i + 1; j < L; ++j) {
      dtensor D = bra[j] * C;
      double v = (D * zket[j]).inner_product(ER[j + 1]) / nrm2;
      szsz[(size_t)i * L + j] = v;
      szsz[(size_t)j * L + i] = v;
      if (j + 1 < L) C = D * psi.A[j];
    }
  }
}

}  // namespace ttb
