"""The work that a user of the two-site DMRG framework has it do, as cases that can be timed.

A DMRG program spends its time in sweeps of two-site updates, and an update in four parts: the
products H_eff*x (three block-sparse contractions through the left environment, the two MPO
tensors and the right environment), the Davidson vector operations between them, the block SVD
with truncation of the two-site tensor, and the environment update.  The cases are

* ``sweep``  -- a whole U(1) sweep of an XXZ chain with random fields through the object API
  (QMPS, QMPO, QDMRG), from a state that the schedule's earlier sweeps have brought to its bond
  dimension, and the magnetisations of the state it leaves;
* ``dense``  -- a whole dense (no quantum numbers) DMRG program, from the product state on;
* ``heff``   -- the products of one Davidson call at one bond, through the contraction ABI, in
  FP64 or in the mixed form (3xTF32 for L*x and *R, FP64 in the middle);
* ``env``    -- one environment update, three contractions;
* ``svd``    -- one block SVD with truncation: density matrices, eigenvalues, the cut on the
  host, eigenvectors of the kept states, the absorbed factor, and the two-site tensor put
  together again from the kept states;
* ``krylov`` -- the vector operations of one Davidson iteration.

Bond dimensions go from the chains' tens to the 3072 of the J1-J2 cylinder.  The charge sectors
of a bond are a discretised Gaussian in 2 Sz with the width measured at bond dimension 3072 on
that cylinder (largest sector about a quarter of the states); MPO links are those of the
nearest-neighbour chain (3 + 1 + 1 states) or of the cylinder (8 + 6 + 6 states).
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensor-tools_b200"))
import tt_b200  # noqa: E402

F64 = torch.float64
CHAIN, CYLINDER = (3, 1), (8, 6)  # MPO link states of charge 0 and of charge +-2 each
SPIN = (-1, 1)                    # 2 Sz of the two states of a site
SIGMA = 3.0                       # width of a bond's charge distribution, in units of 2 Sz


def listed():
    return [
        # a short chain at a small bond dimension: what a first experiment or an early sweep is
        # made of; every kernel is tiny, so launches, synchronisations and host work are the cost
        dict(name="sweep chain L=20 m=32", kind="sweep", L=20, m=32),
        # a production sweep of one of the independent XXZ chains
        dict(name="sweep chain L=48 m=200", kind="sweep", L=48, m=200),
        # the dense path's own configuration: 16 sites, bond dimension 64
        dict(name="dense chain L=16 m=64", kind="dense", L=16, m=64),
        # products at the bond dimension of an early sweep of a chain
        dict(name="heff chain m=128", kind="heff", chi=128, link="chain", mixed=False, nvec=3),
        # the plain FP64 form on the cylinder
        dict(name="heff cylinder m=1400", kind="heff", chi=1400, link="cylinder", mixed=False, nvec=2),
        # the mixed form at a ragged size in the ramp of the schedule
        dict(name="heff mixed m=717", kind="heff", chi=717, link="cylinder", mixed=True, nvec=5),
        # and at the cylinder's full bond dimension: one Davidson call's five products
        dict(name="heff mixed m=3072", kind="heff", chi=3072, link="cylinder", mixed=True, nvec=5),
        # the environment update, FP64 in either form
        dict(name="env cylinder m=2048", kind="env", chi=2048, link="cylinder"),
        # block SVDs of a chain in its ramp, of a chain at its full bond dimension, moving left,
        # and of the cylinder at its full bond dimension
        dict(name="svd m=75", kind="svd", chi=75, right=False),
        dict(name="svd m=512 leftwards", kind="svd", chi=512, right=True),
        dict(name="svd m=3072", kind="svd", chi=3072, right=False),
        # vector operations on a two-site vector of the cylinder's size
        dict(name="krylov n=8000003", kind="krylov", n=8000003, k=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "dense", "heff", "heff", "env", "svd", "svd", "krylov"])
    if kind == "sweep":
        return dict(kind=kind, L=rng.randint(10, 48), m=_log_int(rng, 12, 160))
    if kind == "dense":
        return dict(kind=kind, L=rng.randint(8, 16), m=_log_int(rng, 12, 64))
    if kind == "heff":
        return dict(kind=kind, chi=_log_int(rng, 24, 2400), link=rng.choice(["chain", "cylinder"]),
                    mixed=rng.random() < 0.5, nvec=rng.randint(2, 5))
    if kind == "env":
        return dict(kind=kind, chi=_log_int(rng, 24, 2400), link=rng.choice(["chain", "cylinder"]))
    if kind == "svd":
        return dict(kind=kind, chi=_log_int(rng, 16, 2800), right=rng.random() < 0.5)
    return dict(kind=kind, n=_log_int(rng, 500, 12_000_000), k=rng.randint(1, 6))


# ---- the contraction ABI ---------------------------------------------------------------------
lib = tt_b200.lib
P, I64, D = C.c_void_p, C.c_int64, C.c_double
OUT = np.dtype([("c_off", "i8"), ("m", "i4"), ("n", "i4"), ("ldc", "i4")], align=True)
PAIR = np.dtype([("out_block", "i4"), ("n_m", "i4"), ("n_k", "i4"), ("n_n", "i4"), ("a_off", "i8"), ("b_off", "i8"),
                 ("m_dims", "i4", 6), ("k_dims", "i4", 6), ("n_dims", "i4", 6), ("a_m_stride", "i8", 6),
                 ("a_k_stride", "i8", 6), ("b_k_stride", "i8", 6), ("b_n_stride", "i8", 6)], align=True)
EIG = np.dtype([("g_off", "i8"), ("w_off", "i8"), ("a_off", "i8"), ("n", "i4"), ("flags", "i4")], align=True)
for _name, _args in {
        "tt_contract_plan_keep": [P, P, C.c_int, P, C.c_int, C.c_int, C.c_int, C.POINTER(P)],
        "tt_contract_exec_keep": [P, P, P, P, P, D, C.c_int],
        "tt_plan_release_packed": [P, P], "tt_plan_destroy": [P, P],
        "tt_memcpy_d2h": [P, P, P, C.c_size_t],
        "tt_sym_eigvals_batched": [P, P, C.c_int, P, P, P, P],
        "tt_sym_eigvecs_batched": [P, P, C.c_int, P, P, P, P, P, P, P],
        "tt_vec_ritz_residual_dev": [P, I64, C.c_int, P, P, P, P, P, P],
        "tt_vec_multidot": [P, I64, C.c_int, P, P, P],
        "tt_vec_project_nrm2_dev": [P, I64, C.c_int, P, P, P, P],
        "tt_vec_scal_inv_dev": [P, I64, P, P],
        "tt_qmps_measure_sz": [P, P, P]}.items():
    getattr(lib, _name).restype = C.c_int
    getattr(lib, _name).argtypes = _args

FP64, TF32X3, TF32X3_AUTO = 0, 2, 4
_context = None


def context():
    global _context
    if _context is None:
        _context = tt_b200.Context(0)
    return _context


def call(name, *args):
    if getattr(lib, name)(*args) != 0:
        raise RuntimeError("%s: %s" % (name, lib.tt_get_last_error().decode(errors="replace")))


def at(t):
    return t.ctypes.data if isinstance(t, np.ndarray) else t.data_ptr()


class Layout:
    """Blocks of a block-sparse tensor back to back in one array: key -> (offset, dims)."""

    def __init__(self):
        self.blocks, self.size = {}, 0

    def add(self, key, *dims):
        self.blocks[key] = (self.size, dims)
        self.size += math.prod(dims)

    def random(self, gen, scale=1.0):
        return torch.randn(max(self.size, 2), dtype=F64, device="cuda", generator=gen) * scale


class Contraction:
    """Output blocks and block pairs of one contraction, and the plan made of them."""

    def __init__(self):
        self.outs, self.pairs, self.handle, self.flops = [], [], None, 0.0

    def out(self, off, m, n):
        self.outs.append((off, m, n, m))
        return len(self.outs) - 1

    def pair(self, o, a_off, b_off, m, k, n):
        """m: [(dim, stride in A)], k: [(dim, stride in A, stride in B)], n: [(dim, stride in B)]; first mode fastest."""
        pad = lambda v: list(v) + [0] * (6 - len(v))  # noqa: E731
        self.pairs.append((o, len(m), len(k), len(n), a_off, b_off, pad([x[0] for x in m]),
                           pad([x[0] for x in k]), pad([x[0] for x in n]), pad([x[1] for x in m]), pad([x[1] for x in k]),
                           pad([x[2] for x in k]), pad([x[1] for x in n])))
        self.flops += 2.0 * math.prod(x[0] for x in m) * math.prod(x[0] for x in k) * math.prod(x[0] for x in n)

    def arrays(self):
        return np.array(self.outs, dtype=OUT), np.array(self.pairs, dtype=PAIR)

    def plan(self, precision=FP64, keep=0):
        self.handle = make_plan(*self.arrays(), precision, keep)
        return self

    def exec(self, a, b, c, keep=0):
        call("tt_contract_exec_keep", context().h, self.handle, at(a), at(b), at(c), 1.0, keep)

    def release(self):
        call("tt_plan_release_packed", context().h, self.handle)

    def __del__(self):
        if self.handle:
            lib.tt_plan_destroy(context().h, self.handle)


def make_plan(outs, pairs, precision=FP64, keep=0):
    h = P()
    call("tt_contract_plan_keep", context().h, at(outs), len(outs), at(pairs), len(pairs), precision, keep, C.byref(h))
    return h


def exact_contraction(con, a, b, size):
    """The contraction in plain torch, pair by pair over strided views."""
    c = torch.zeros(max(size, 2), dtype=F64, device="cuda")
    for o, nm, nk, nn, ao, bo, md, kd, nd, am, ak, bk, bn in con.pairs:
        rev = lambda v, n: tuple(v[:n][::-1])  # noqa: E731
        M, K, N = math.prod(md[:nm]), math.prod(kd[:nk]), math.prod(nd[:nn])
        A = a.as_strided(rev(kd, nk) + rev(md, nm), rev(ak, nk) + rev(am, nm), ao).reshape(K, M)
        B = b.as_strided(rev(nd, nn) + rev(kd, nk), rev(bn, nn) + rev(bk, nk), bo).reshape(N, K)
        off, m, n, ld = con.outs[o]
        c.as_strided((n, m), (ld, 1), off).addmm_(B, A)
    return c


def bond(chi, parity):
    """Charge sectors {2 Sz: states} of a bond of `chi` states."""
    qs = [q for q in range(-40, 41) if (q - parity) % 2 == 0]
    w = {q: math.exp(-q * q / (2 * SIGMA * SIGMA)) for q in qs}
    tot = sum(w.values())
    return {q: max(1, round(chi * w[q] / tot)) for q in qs if chi * w[q] / tot >= 0.5}


def link(kind):
    w0, w2 = CHAIN if kind == "chain" else CYLINDER
    return {-2: w2, 0: w0, 2: w2}


def mpo_values(layout, gen):
    """Entries of an MPO tensor: mostly zeros, else couplings."""
    u = torch.rand(max(layout.size, 2), dtype=F64, device="cuda", generator=gen)
    v = torch.where(u < 0.05, 0.5 + 0 * u, 0 * u)
    return torch.where(u > 0.9, 2.0 * u - 0.9, v)


class Heff:
    """H_eff*x at a bond in the middle: L[a',w,a] x[a,s1,s2,b] M[w,s1,s2;s1',s2',w'] R[b',w',b]."""

    def __init__(self, chi, kind):
        a, b, w = bond(chi, 0), bond(chi, 0), link(kind)
        self.L, self.x, self.M, self.R, self.T1, self.T2, self.y = (Layout() for _ in range(7))
        two = [(s, t) for t in SPIN for s in SPIN]
        for qa in a:
            for qw in w:
                if qa + qw in a:
                    self.L.add((qa + qw, qw, qa), a[qa + qw], w[qw], a[qa])
        for qb in b:
            for qw in w:
                if qb + qw in b:
                    self.R.add((qb + qw, qw, qb), b[qb + qw], w[qw], b[qb])
        for qa in a:
            for s, t in two:
                if qa + s + t in b:
                    self.x.add((qa, s, t, qa + s + t), a[qa], b[qa + s + t])
                    self.y.add((qa, s, t, qa + s + t), a[qa], b[qa + s + t])
        for qw in w:
            for s, t in two:
                for u, v in two:
                    if qw + u + v - s - t in w:
                        self.M.add((qw, s, t, u, v), w[qw], w[qw + u + v - s - t])
        self.c1, self.c2, self.c3 = Contraction(), Contraction(), Contraction()
        for (qp, qw, qa), (lo, (dp, dw, da)) in self.L.blocks.items():
            for s, t in two:
                if (qa, s, t, qa + s + t) in self.x.blocks:
                    xo, (_, db) = self.x.blocks[qa, s, t, qa + s + t]
                    self.T1.add((qp, qw, s, t, qa + s + t), dp, dw, db)
                    o = self.c1.out(self.T1.blocks[qp, qw, s, t, qa + s + t][0], dp * dw, db)
                    self.c1.pair(o, lo, xo, [(dp * dw, 1)], [(da, dp * dw, 1)], [(db, da)])
        outs = {}
        for (qp, qw, s, t, qb), (to, (dp, dw, db)) in self.T1.blocks.items():
            for u, v in two:
                if (qw, s, t, u, v) not in self.M.blocks:
                    continue
                qv = qw + u + v - s - t
                mo, (_, dv) = self.M.blocks[qw, s, t, u, v]
                key = (qp, u, v, qv, qb)
                if key not in outs:
                    self.T2.add(key, dp, db, dv)
                    outs[key] = self.c2.out(self.T2.blocks[key][0], dp * db, dv)
                self.c2.pair(outs[key], to, mo, [(dp, 1), (db, dp * dw)], [(dw, dp, 1)], [(dv, dw)])
        for (qp, u, v, qf), (yo, (dp, df)) in self.y.blocks.items():
            o = self.c3.out(yo, dp, df)
            for qv in w:
                key, rk = (qp, u, v, qv, qf - qv), (qf, qv, qf - qv)
                if key in self.T2.blocks and rk in self.R.blocks:
                    to, (_, db, dv) = self.T2.blocks[key]
                    self.c3.pair(o, to, self.R.blocks[rk][0], [(dp, 1)], [(db, dp, df * dv), (dv, dp * db, df)], [(df, 1)])


class Env:
    """One environment update: E[a',w,a], site tensor A[a,s,b], MPO tensor W[w,s';s,w2] -> E[b',w2,b]."""

    def __init__(self, chi, kind):
        a, b, w = bond(chi, 0), bond(chi, 1), link(kind)
        self.E, self.A, self.W, self.T4, self.T5, self.F = (Layout() for _ in range(6))
        for qa in a:
            for qw in w:
                if qa + qw in a:
                    self.E.add((qa + qw, qw, qa), a[qa + qw], w[qw], a[qa])
            for s in SPIN:
                if qa + s in b:
                    self.A.add((qa, s, qa + s), a[qa], b[qa + s])
        for qw in w:
            for u in SPIN:
                for s in SPIN:
                    if qw + u - s in w:
                        self.W.add((qw, u, s), w[qw], w[qw + u - s])
        self.c1, self.c2, self.c3 = Contraction(), Contraction(), Contraction()
        for (qp, qw, qa), (eo, (dp, dw, da)) in self.E.blocks.items():
            for u in SPIN:
                if (qp, u, qp + u) in self.A.blocks:
                    ao, (_, dg) = self.A.blocks[qp, u, qp + u]
                    self.T4.add((u, qp + u, qw, qa), dg, dw, da)
                    o = self.c1.out(self.T4.blocks[u, qp + u, qw, qa][0], dg, dw * da)
                    self.c1.pair(o, ao, eo, [(dg, dp)], [(dp, 1, 1)], [(dw * da, dp)])
        outs = {}
        for (u, qg, qw, qa), (to, (dg, dw, da)) in self.T4.blocks.items():
            for s in SPIN:
                if (qw, u, s) not in self.W.blocks or (qa, s, qa + s) not in self.A.blocks:
                    continue
                wo, (_, dv) = self.W.blocks[qw, u, s]
                key = (qg, qa, s, qw + u - s)
                if key not in outs:
                    self.T5.add(key, dg, da, dv)
                    outs[key] = self.c2.out(self.T5.blocks[key][0], dg * da, dv)
                self.c2.pair(outs[key], to, wo, [(dg, 1), (da, dg * dw)], [(dw, dg, 1)], [(dv, dw)])
        outs = {}
        for (qg, qa, s, qv), (to, (dg, da, dv)) in self.T5.blocks.items():
            ao, (_, db) = self.A.blocks[qa, s, qa + s]
            key = (qg, qv, qa + s)
            if key not in outs:
                self.F.add(key, dg, dv, db)
                outs[key] = self.c3.out(self.F.blocks[key][0], dg * dv, db)
            self.c3.pair(outs[key], to, ao, [(dg, 1), (dv, dg * da)], [(da, dg, 1)], [(db, da)])


class Svd:
    """The block SVD of a two-site tensor x[a,s1,s2,b] between (a,s1) and (s2,b), to chi states."""

    def __init__(self, chi, right):
        a, b, mid = bond(chi, 0), bond(chi, 0), bond(2 * chi, 1)
        self.chi, self.right, self.x, self.sectors = chi, right, Layout(), []
        for qa in a:
            for s in SPIN:
                for t in SPIN:
                    if qa + s + t in b:
                        self.x.add((qa, s, t), a[qa], b[qa + s + t])
        g_off = w_off = 0
        for q in sorted(set(qa + s for qa, s, _ in self.x.blocks)):
            rows = [(q - s, s) for s in SPIN if q - s in a]
            cols = [(q + t, t) for t in SPIN if q + t in b]
            if not rows or not cols:
                continue
            dr, dc = [a[r[0]] for r in rows], [b[c[0]] for c in cols]
            g = sum(dc) if right else sum(dr)
            self.sectors.append(dict(q=q, rows=rows, cols=cols, dr=dr, dc=dc, g=g, g_off=g_off, w_off=w_off,
                                     weight=math.exp(-q * q / (2 * SIGMA * SIGMA)), scale=mid.get(q, 1) / 2))
            g_off, w_off = g_off + g * g, w_off + g
        self.gtot, self.wtot = g_off, w_off
        self.gram, self.absorb, self.join = Contraction(), Contraction(), Contraction()
        self.probs = np.array([(s["g_off"], s["w_off"], 0, s["g"], 0) for s in self.sectors], dtype=EIG)
        sec_of_absorb, sec_of_join = [], []
        for k, s in enumerate(self.sectors):
            kept, other = ("cols", "rows") if right else ("rows", "cols")
            kd, od = (s["dc"], s["dr"]) if right else (s["dr"], s["dc"])
            off = [sum(kd[:i]) for i in range(len(kd))]
            for i in range(len(kd)):
                for j in range(len(kd)):
                    o = self.gram.out(s["g_off"] + off[i] + s["g"] * off[j], kd[i], kd[j])
                    self.gram.outs[o] = self.gram.outs[o][:3] + (s["g"],)
                    for r in range(len(od)):
                        bi, bj = self.block(s, i, r), self.block(s, j, r)
                        self.gram.pair(o, bi[0], bj[0], [(kd[i], bi[1])], [(od[r], bi[2], bj[2])], [(kd[j], bj[1])])
            for r in range(len(od)):
                o = self.absorb.out(0, 0, 0)
                sec_of_absorb.append((k, od[r]))
                for i in range(len(kd)):
                    bi = self.block(s, i, r)
                    if right:  # U(l) = sum_j x(l, r_j) Z_j
                        self.absorb.pair(o, bi[0], s["g_off"] + off[i], [(od[r], bi[2])], [(kd[i], bi[1], 1)], [(1, s["g"])])
                    else:      # V(r) = sum_i Z_i^T x(l_i, r)
                        self.absorb.pair(o, s["g_off"] + off[i], bi[0], [(1, s["g"])], [(kd[i], 1, bi[1])], [(od[r], bi[2])])
                    jo = self.join.out(bi[0], *((od[r], kd[i]) if right else (kd[i], od[r])))
                    sec_of_join.append((k, o))
                    if right:  # x(l, r_j) = U(l) Z_j^T
                        self.join.pair(jo, 0, s["g_off"] + off[i], [(od[r], 1)], [(1, od[r], s["g"])], [(kd[i], 1)])
                    else:      # x(l_i, r) = Z_i V(r)
                        self.join.pair(jo, s["g_off"] + off[i], 0, [(kd[i], 1)], [(1, s["g"], 1)], [(od[r], 1)])
        self.absorb_sec = np.array([k for k, _ in sec_of_absorb])
        self.absorb_dim = np.array([d for _, d in sec_of_absorb])
        self.join_sec = np.array([k for k, _ in sec_of_join])
        self.join_src = np.array([o for _, o in sec_of_join])
        self.limit = np.array([min(sum(s["dr"]), sum(s["dc"])) for s in self.sectors])

    def block(self, s, i, r):
        """Block of kept-side tuple i and other-side tuple r: offset, stride along the kept side, along the other."""
        l, c = (r, i) if self.right else (i, r)
        off, (da, _) = self.x.blocks[s["rows"][l][0], s["rows"][l][1], s["cols"][c][1]]
        return (off, da, 1) if self.right else (off, 1, da)

    def values(self, gen):
        """A two-site tensor whose singular values fall off in every sector as those of a ground state do: to about
        1e-9 of the weight at the states that the cut drops first."""
        x = torch.zeros(self.x.size, dtype=F64, device="cuda")
        for s in self.sectors:
            nr, nc = sum(s["dr"]), sum(s["dc"])
            r = min(nr, nc)
            u, _ = torch.linalg.qr(torch.randn(nr, r, dtype=F64, device="cuda", generator=gen))
            v, _ = torch.linalg.qr(torch.randn(nc, r, dtype=F64, device="cuda", generator=gen))
            j = torch.arange(r, dtype=F64, device="cuda")
            lam = torch.exp(-20.0 * j / max(s["scale"], 4.0)) * (0.8 + 0.4 * torch.rand(r, dtype=F64, device="cuda", generator=gen))
            m = (u * (s["weight"] * lam).sqrt()) @ v.T
            for i, (qa, sa) in enumerate(s["rows"]):
                for k, (_, t) in enumerate(s["cols"]):
                    off, (da, db) = self.x.blocks[qa, sa, t]
                    r0, c0 = sum(s["dr"][:i]), sum(s["dc"][:k])
                    x[off:off + da * db] = m[r0:r0 + da, c0:c0 + db].T.reshape(-1)
        return x / x.norm()

    def cut(self, w):
        """Kept states per sector: the chi largest of all sectors' eigenvalues (ties by sector and position)."""
        lam = np.concatenate([np.abs(w[s["w_off"]:s["w_off"] + n]) for s, n in zip(self.sectors, self.limit)])
        sec = np.repeat(np.arange(len(self.sectors)), self.limit)
        return np.bincount(sec[np.argsort(-lam, kind="stable")[:self.chi]], minlength=len(self.sectors)).astype(np.int32)

    def absorb_arrays(self, nv):
        """Output blocks and pairs of the absorbed factor and of the joined tensor for nv kept states per sector."""
        outs, pairs = self.absorb_np
        outs, pairs = outs.copy(), pairs.copy()
        nd = nv[self.absorb_sec]
        outs["m"], outs["n"] = (self.absorb_dim, nd) if self.right else (nd, self.absorb_dim)
        outs["ldc"] = outs["m"]
        size = outs["m"].astype(np.int64) * outs["n"]
        outs["c_off"] = np.cumsum(size) - size
        pairs["n_dims" if self.right else "m_dims"][:, 0] = nd[pairs["out_block"]]
        jouts, jpairs = self.join_np
        jpairs = jpairs.copy()
        jnd = nv[self.join_sec]
        jpairs["k_dims"][:, 0] = jnd
        src = outs["c_off"][self.join_src]
        if self.right:
            jpairs["a_off"] = src
        else:
            jpairs["b_off"] = src
            jpairs["b_n_stride"][:, 0] = jnd
        live = (outs["m"] > 0) & (outs["n"] > 0)
        if not live.all():  # sectors that keep nothing have no factor
            new = np.cumsum(live) - 1
            pairs = pairs[live[pairs["out_block"]]]
            pairs["out_block"] = new[pairs["out_block"]]
            outs = outs[live]
            jpairs = jpairs[jnd > 0]
        return outs, pairs, jouts, jpairs, int(size.sum())


# ---- the cases ---------------------------------------------------------------------------------
def chain_hamiltonian(L, seed):
    """An XXZ chain with random anisotropy and small random fields, as the independent-chains workload has them."""
    r = np.random.default_rng(seed)
    delta, h = float(r.uniform(0.5, 1.5)), r.uniform(-0.1, 0.1, L)
    ampo = tt_b200.AutoMPO()
    for i in range(L - 1):
        ampo.add(0.5, "S+", i, "S-", i + 1).add(0.5, "S-", i, "S+", i + 1).add(delta, "Sz", i, "Sz", i + 1)
    for i in range(L):
        ampo.add(float(h[i]), "Sz", i)
    return ampo


def prepare(case, seed):
    context()
    tt_b200.set_precision()
    kind, st = case["kind"], dict(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind == "sweep":
        L, m = case["L"], case["m"]
        st["psi"] = tt_b200.QMPS(L, [i % 2 for i in range(L)])
        st["H"] = tt_b200.QMPO.from_autompo(chain_hamiltonian(L, seed), L)
        st["run"] = tt_b200.QDMRG(st["psi"], st["H"])
        for mm in (max(8, m // 4), max(8, m // 2), m, m):
            st["run"].sweep(mm, 1e-10, 6)
    elif kind == "dense":
        st["H"] = tt_b200.DMPO.from_autompo(chain_hamiltonian(case["L"], seed), case["L"])
    elif kind == "heff":
        h = st["op"] = Heff(case["chi"], case["link"])
        st["L"], st["R"] = h.L.random(gen, case["chi"] ** -0.5), h.R.random(gen, case["chi"] ** -0.5)
        st["M"] = mpo_values(h.M, gen)
        st["x"] = [h.x.random(gen, h.x.size ** -0.5) for _ in range(case["nvec"])]
        st["T1"], st["T2"] = torch.empty(h.T1.size, dtype=F64, device="cuda"), torch.empty(h.T2.size, dtype=F64, device="cuda")
        st["y"] = [torch.empty(h.y.size, dtype=F64, device="cuda") for _ in range(case["nvec"])]
        # the mixed form's choice per contraction: tensor cores where there is work for them, FP64 in the middle
        prec = lambda c: FP64 if not case["mixed"] else TF32X3 if c.flops >= 2e10 else TF32X3_AUTO  # noqa: E731
        h.c1.plan(prec(h.c1), 1), h.c2.plan(), h.c3.plan(prec(h.c3), 2)
    elif kind == "env":
        e = st["op"] = Env(case["chi"], case["link"])
        st["E"], st["W"] = e.E.random(gen, case["chi"] ** -0.5), mpo_values(e.W, gen)
        st["A"] = e.A.random(gen, case["chi"] ** -0.5)
        st["T4"], st["T5"], st["F"] = (torch.empty(t.size, dtype=F64, device="cuda") for t in (e.T4, e.T5, e.F))
        for c in (e.c1, e.c2, e.c3):
            c.plan()
    elif kind == "svd":
        s = st["op"] = Svd(case["chi"], case["right"])
        s.gram_np, s.absorb_np, s.join_np = s.gram.arrays(), s.absorb.arrays(), s.join.arrays()
        st["x"] = s.values(gen)
        st["G"], st["Z"] = (torch.empty(s.gtot, dtype=F64, device="cuda") for _ in range(2))
        st["W"], st["T"] = (torch.empty(n, dtype=F64, device="cuda") for n in (s.wtot, 3 * s.wtot))
        st["work"] = torch.empty(3 * s.gtot, dtype=F64, device="cuda")
        st["V"] = torch.empty(max(2, sum(int(g["g"]) * max(sum(g["dr"]), sum(g["dc"])) for g in s.sectors)), dtype=F64, device="cuda")
        st["theta"], st["w"] = torch.empty_like(st["x"]), np.empty(s.wtot)
    else:
        n, k = case["n"], case["k"]
        v = torch.randn(k, n + (n & 1), dtype=F64, device="cuda", generator=gen)
        v[:, n:] = 0
        v = torch.linalg.qr(v.T)[0].T.contiguous()
        st["v"], st["va"] = list(v), list(torch.randn(k, n + (n & 1), dtype=F64, device="cuda", generator=gen) * n ** -0.5)
        c = torch.randn(2 * k + 1, dtype=F64, device="cuda", generator=gen)
        st["cx"], st["cq"] = c[:k] / c[:k].norm(), c[k:].clone()
        st["xr"], st["q"], st["s"] = torch.zeros(n, dtype=F64, device="cuda"), torch.zeros(n, dtype=F64, device="cuda"), torch.zeros(64, dtype=F64, device="cuda")
        st["pv"], st["pva"] = ((P * (k + 1))(*[t.data_ptr() for t in w + [st["q"]]]) for w in (st["v"], st["va"]))
    torch.cuda.synchronize()
    return st


def run(st):
    kind, h = st["kind"], context().h
    if kind == "sweep":
        energy = st["run"].sweep(st["m"], 1e-10, 6)
        sz = np.zeros(st["L"])
        call("tt_qmps_measure_sz", st["psi"].h, sz.ctypes.data, None)
        return {"energy": energy, "sz": sz}
    if kind == "dense":
        psi = tt_b200.DMPS(st["L"], [i % 2 for i in range(st["L"])])
        energy, sweeps, _ = tt_b200.ddmrg_run(psi, st["H"], 3, [max(8, st["m"] // 2), st["m"], st["m"]], [1e-10], [4])
        return {"energy": energy, "sweeps": sweeps}
    if kind == "heff":
        op = st["op"]
        # L and R are fixed through a Davidson call: their packed form is kept for its products and given back at its end
        for x, y in zip(st["x"], st["y"]):
            op.c1.exec(st["L"], x, st["T1"], 1 | 8)
            op.c2.exec(st["T1"], st["M"], st["T2"])
            op.c3.exec(st["T2"], st["R"], y, 2 | 4)
        op.c1.release(), op.c3.release()
        return {"y": st["y"]}
    if kind == "env":
        op = st["op"]
        op.c1.exec(st["A"], st["E"], st["T4"])
        op.c2.exec(st["T4"], st["W"], st["T5"])
        op.c3.exec(st["T5"], st["A"], st["F"])
        return {"E": st["F"]}
    if kind == "svd":
        op, x = st["op"], st["x"]

        def once(outs, pairs, a, b, c):  # kept counts change from step to step: a plan of its own each time
            p = make_plan(outs, pairs)
            call("tt_contract_exec_keep", h, p, at(a), at(b), at(c), 1.0, 0)
            call("tt_plan_destroy", h, p)

        once(*op.gram_np, x, x, st["G"])
        call("tt_sym_eigvals_batched", h, at(op.probs), len(op.probs), at(st["G"]), at(st["T"]), at(st["W"]), None)
        call("tt_memcpy_d2h", h, at(st["w"]), at(st["W"]), 8 * op.wtot)
        nv = op.cut(st["w"])
        call("tt_sym_eigvecs_batched", h, at(op.probs), len(op.probs), at(nv), at(st["G"]), at(st["T"]), at(st["W"]),
             at(st["Z"]), at(st["work"]), None)
        outs, pairs, jouts, jpairs, _ = op.absorb_arrays(nv)
        a, b = (x, st["Z"]) if op.right else (st["Z"], x)
        once(outs, pairs, a, b, st["V"])
        a, b = (st["V"], st["Z"]) if op.right else (st["Z"], st["V"])
        once(jouts, jpairs, a, b, st["theta"])
        return {"eigenvalues": st["W"], "theta": st["theta"], "kept": nv}
    n, k, s = st["n"], st["k"], st["s"]
    q, slot = at(st["q"]), lambda i: at(s) + 8 * i  # noqa: E731
    call("tt_vec_ritz_residual_dev", h, n, k, st["pv"], st["pva"], at(st["cx"]), at(st["cq"]), at(st["xr"]), q)
    call("tt_vec_nrm2", h, n, q, slot(40))
    call("tt_vec_multidot", h, n, k, st["pv"], q, slot(0))
    call("tt_vec_project_nrm2_dev", h, n, k, st["pv"], slot(0), q, slot(41))
    call("tt_vec_scal_inv_dev", h, n, slot(41), q)
    call("tt_vec_multidot", h, n, k + 1, st["pv"], at(st["va"][0]), slot(16))
    return {"ritz": st["xr"], "new": st["q"], "overlaps": s[:k], "row": s[16:17 + k], "norms": s[40:42]}


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "dense"):
        L, m = case["L"], case["m"]
        flops = data = 0.0
        for i in range(1, L):
            d = float(min(m, 2 ** min(i, L - i)))
            fill = 1.0 if kind == "dense" else 0.2
            per = fill * (5 * (2 * 5 * 4 * 2 * d ** 3) + 2 * 5 * 2 * 2 * 2 * d ** 3) + 30 * fill * fill * d ** 3
            flops += 2 * per
            data += 2 * 8 * (2 * 5 * d * d + 2 * 4 * d * d)
        n = 3 if kind == "dense" else 1
        return {"bytes": n * data, "flops": n * flops}
    if kind == "heff":
        h = Heff(case["chi"], case["link"])
        return {"bytes": 8.0 * (h.L.size + h.R.size + h.M.size + case["nvec"] * 2 * h.x.size),
                "flops": case["nvec"] * (h.c1.flops + h.c2.flops + h.c3.flops)}
    if kind == "env":
        e = Env(case["chi"], case["link"])
        return {"bytes": 8.0 * (e.E.size + e.A.size + e.W.size + e.F.size), "flops": e.c1.flops + e.c2.flops + e.c3.flops}
    if kind == "svd":
        s = Svd(case["chi"], case["right"])
        flops = s.gram.flops / 2
        for t in s.sectors:
            g, o = t["g"], sum(t["dr"]) if case["right"] else sum(t["dc"])
            flops += 4 / 3 * g ** 3 + 2.0 * g * g * (g / 2) + 4.0 * g * o * (g / 2)
        return {"bytes": 8.0 * (2 * s.x.size + s.wtot), "flops": flops}
    n, k = case["n"], case["k"]
    # the k basis vectors and products read once, the Ritz vector and the new vector written once
    return {"bytes": 8.0 * n * (2 * k + 2), "flops": 2.0 * n * (2 * k + 1 + k + k + 1 + 2)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sweep", "dense"):
        return None
    st = prepare(case, seed)
    if kind == "heff":
        h, ys = st["op"], []
        for x in st["x"]:
            t1 = exact_contraction(h.c1, st["L"], x, h.T1.size)
            t2 = exact_contraction(h.c2, t1, st["M"], h.T2.size)
            ys.append(exact_contraction(h.c3, t2, st["R"], h.y.size))
        return {"y": ys}
    if kind == "env":
        e = st["op"]
        t4 = exact_contraction(e.c1, st["A"], st["E"], e.T4.size)
        t5 = exact_contraction(e.c2, t4, st["W"], e.T5.size)
        return {"E": exact_contraction(e.c3, t5, st["A"], e.F.size)}
    if kind == "svd":
        op, x, vecs = st["op"], st["x"], []
        w, theta = np.empty(op.wtot), torch.empty_like(st["x"])
        for s in op.sectors:
            m = torch.cat([torch.cat([x[op.x.blocks[qa, sa, t][0]:][:da * db].reshape(db, da).T for db, (_, t) in zip(s["dc"], s["cols"])], 1)
                           for da, (qa, sa) in zip(s["dr"], s["rows"])], 0)
            lam, z = torch.linalg.eigh(m.T @ m if op.right else m @ m.T)
            w[s["w_off"]:s["w_off"] + s["g"]] = lam.flip(0).cpu().numpy()
            vecs.append((m, z.flip(1)))
        nv = op.cut(w)
        for s, (m, z), n in zip(op.sectors, vecs, nv):
            z = z[:, :n]
            m = (m @ z) @ z.T if op.right else z @ (z.T @ m)
            for i, (qa, sa) in enumerate(s["rows"]):
                for k, (_, t) in enumerate(s["cols"]):
                    off, (da, db) = op.x.blocks[qa, sa, t]
                    r0, c0 = sum(s["dr"][:i]), sum(s["dc"][:k])
                    theta[off:off + da * db] = m[r0:r0 + da, c0:c0 + db].T.reshape(-1)
        return {"eigenvalues": w, "theta": theta, "kept": nv}
    n, k = case["n"], case["k"]
    v, va = [t[:n] for t in st["v"]], [t[:n] for t in st["va"]]
    ritz = sum(st["cx"][j] * v[j] for j in range(k))
    q = sum(st["cq"][j] * va[j] for j in range(k)) + st["cq"][k] * ritz
    overlaps = torch.stack([t @ q for t in v])
    new = q - sum(overlaps[j] * v[j] for j in range(k))
    norms = torch.stack([q.norm(), new.norm()])
    new = new / norms[1]
    return {"ritz": ritz, "new": new, "overlaps": overlaps, "row": torch.stack([t @ va[0] for t in v + [new]]), "norms": norms}
