#!/usr/bin/env python
"""Benchmark of the B200 two-site DMRG inner loop.

Default workload (the J1-J2 cylinder configuration): U(1)-conserving two-site
DMRG of the spin-1/2 J1-J2 Heisenberg model, J1 = 1, J2 = 0.5, on a 6 x 16
cylinder (periodic around the 6-site circumference, 96 sites numbered in snake
order), total Sz = 0 from the Neel state, SVD cutoff 1e-10, Davidson at most
4 iterations (the reference's hard-wired tolerance 1e-12), bond dimension
3072.

Set-up (untimed): the ramp maxdim 64, 128, 256, 512, 1024, 2048 with noise
1e-6 decaying linearly to 0 over those six sweeps, then one sweep at 3072
without noise, all in the chosen (mixed-precision) form; the state is
checkpointed.  Each precision then loads the same checkpoint, builds its
environments and moves the orthogonality centre to the middle of the chain
(untimed).  A step is a fixed block of mid-chain two-site updates at bond
dimension 3072: four left-to-right updates over sites 46..49 and four
right-to-left updates back (8 updates, each Davidson + block SVD + environment
update).  W warm-up and K timed steps per precision, CUDA events on the
library's stream, L2 flushed before every step (the environments alone are
tens of GB, far larger than L2).

Reported value: seconds per sweep-equivalent of the chosen form (TF32 / 3xTF32
on tcgen05 for the contractions its cost model picks, FP64 everywhere else):
the mean time per timed two-site update times the 190 updates of a sweep
(2 x 95 bonds) -- every update timed is at the full bond dimension, so this
is the cost of a sweep at bond dimension 3072 throughout; ``ms_per_step`` is
the measured time of one block step.  ``full_sweep`` holds a measured full
sweep per precision (its edge bonds are smaller).  ``fp64`` is the plain GPU
form on the same schedule; ``mixed`` repeats the chosen form's numbers with
|dE|/N against FP64, both energies being <psi|H|psi>/<psi|psi> contracted in
FP64 after identical schedules.  Rooflines: H_eff*x algorithmic TFLOP/s
(event-timed product launches) against the cuBLAS DGEMM peak (FP64) and the
cuBLAS TF32 peak (mixed; a 3xTF32 flop costs three TF32 products), both
measured in this run.  ``e2e`` repeats steps of the chosen form through the
public C ABI with the block's MPS site tensors uploaded from pinned host
memory before and downloaded after every step.

Other workloads (``--workload``): ``heisenberg`` -- the L = 100 Heisenberg
chain to maxdim 512 (a step is one full sweep); ``gemm`` -- single-block
contraction throughput per precision; ``xxz-chains`` -- independent chains
sharing one GPU.

``--impl reference`` times the CPU restatement of the reference algorithm
(oracle/, numpy + LAPACK on all host cores) on the same workload: real
two-site updates (Davidson, block SVD, environment update) at bond dimension
3072 in the middle of the 96-site cylinder, on environments contracted with
the same MPO through a state that is the Neel product state outside a 12-site
window on each side and random left/right-canonical isometries (growing the
bond to 3072) inside.  One update costs tens of seconds on the host, so the
number of timed updates is capped by --ref-budget seconds (reported).
"""
from __future__ import annotations

import argparse
import json
import os
import resource
import shutil
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "tensor-tools_b200")
sys.path.insert(0, PKG)
sys.path.insert(0, ROOT)

METRIC = "sec/sweep & H_eff*x TFLOP/s: TF32/FP32 grouped vs FP64 GPU at |dE|/N<=1e-8"

# the J1-J2 cylinder configuration
C5 = dict(Nx=16, Ny=6, J2=0.5, maxdim=3072, cutoff=1e-10, max_restart=4,
          ramp=[64, 128, 256, 512, 1024, 2048], noise0=1e-6, block=4)
C5_N = C5["Nx"] * C5["Ny"]
C5_MID = C5_N // 2 - C5["block"] // 2          # 46: the block spans sites 46..50
C5_UPDATES_PER_SWEEP = 2 * (C5_N - 1)           # 190
CHOSEN = "tf32x3-auto"
# the environment updates stay in FP64 in the chosen form: FP64 environments
# keep the Ritz values free of a first-order bias.  Measured on this workload
# with --env-prec tf32x3-auto: 6% less time per sweep, but |dE|/N = 1.1e-8
# against FP64 after a full sweep at bond dimension 3072 (2.4e-9 with FP64
# environments), above the 1e-8 the mixed form must hold.
ENV_PREC = "fp64"


def c5_ramp(args):
    """The ramp's bond dimensions below the workload's (a smaller --maxdim,
    e.g. for a profiler capture, stops the ramp early)."""
    return [m for m in C5["ramp"] if m < args.maxdim]


def c5_config(args):
    return {
        "workload": "U(1) two-site DMRG, spin-1/2 J1-J2 Heisenberg (J1=1, J2=0.5) on the 6x16 cylinder "
                    "(periodic y, 96 sites, snake order), Sz=0 Neel start, maxdim %d, cutoff 1e-10, "
                    "Davidson max %d iters (tol 1e-12 as hard-wired in the reference)" % (args.maxdim,
                                                                                           args.max_restart),
        "L": C5_N, "maxdim": args.maxdim, "cutoff": C5["cutoff"], "max_restart": args.max_restart,
        "setup": "untimed ramp maxdim %s with noise 1e-6 -> 0 over those sweeps, one sweep at maxdim %d, "
                 "checkpoint; per precision: load, buildEnv, centre to site %d" % (c5_ramp(args), args.maxdim, C5_MID),
        "step": "%d two-site updates at maxdim %d: left-to-right over sites %d..%d and back" % (
            2 * args.block, args.maxdim, C5_MID, C5_MID + args.block - 1),
        "value_definition": "mean seconds per timed two-site update x %d updates per sweep" % C5_UPDATES_PER_SWEEP,
        "l2": "environments (tens of GB) far larger than L2; L2 flushed before every step",
        "davidson_tol": 1e-12,
    }


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=3)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--workload", default="j1j2", choices=["j1j2", "heisenberg", "xxz-chains", "gemm"])
    p.add_argument("--maxdim", type=int, default=C5["maxdim"])
    p.add_argument("--max-restart", type=int, default=C5["max_restart"])
    p.add_argument("--block", type=int, default=C5["block"])
    p.add_argument("--e2e-steps", type=int, default=2)
    p.add_argument("--cpu-budget", type=float, default=30.0, help="seconds of CPU baseline sampling (rank 0)")
    p.add_argument("--ref-budget", type=float, default=900.0,
                   help="seconds of warm-up and timed updates of the reference arm")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-full-sweep", action="store_true")
    p.add_argument("--breakdown", action="store_true", help="one further step per precision with phase times")
    p.add_argument("--env-prec", default=ENV_PREC, help="environment-update precision of the chosen form")
    p.add_argument("--no-clock-sampler", action="store_true", help="diagnostic: no nvidia-smi sampling")
    p.add_argument("--detail", help="file for the whole result: per-step times, phases and host load of both arms")
    p.add_argument("--gemm-size", type=int, default=4096)
    p.add_argument("--precisions", default="fp64,tf32x3,tf32")
    p.add_argument("--chains", type=int, default=64)
    p.add_argument("--chain-sweeps", type=int, default=8)
    p.add_argument("--streams", type=int, default=16)
    return p.parse_args()


# ---------------------------------------------------------------------------
# clocks sampled while the timed region runs
# ---------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def start(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.FIELDS,
                                       "--format=csv,noheader,nounits", "-lms", "200"],
                                      stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None

    def stop(self):
        if self.p is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.p.terminate()
        self.p.wait(timeout=10)
        self.f.flush()
        rows = [r.split(",") for r in open(self.f.name).read().strip().splitlines() if r.count(",") >= 8]
        os.unlink(self.f.name)
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in rows:
            for k, nm in enumerate(names):
                if "Active" in r[5 + k] and "Not" not in r[5 + k]:
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(rows)}


def load_hbm_peak():
    """The measured HBM copy bandwidth (GB/s) of this pool's B200s, if present."""
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"])
    except (OSError, KeyError, ValueError):
        return None


def measured_peaks(torch):
    """cuBLAS DGEMM (FP64 tensor path) and TF32 GEMM throughput, 8192^3, best of 3."""
    n = 8192
    out = {}
    prev = torch.backends.cuda.matmul.allow_tf32
    for name, dt, tf32 in (("fp64", torch.float64, False), ("tf32", torch.float32, True)):
        torch.backends.cuda.matmul.allow_tf32 = tf32
        a = torch.randn(n, n, dtype=dt, device="cuda")
        b = torch.randn(n, n, dtype=dt, device="cuda")
        for _ in range(2):
            torch.matmul(a, b)
        torch.cuda.synchronize()
        best = 0.0
        for _ in range(3):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            torch.matmul(a, b)
            e1.record()
            torch.cuda.synchronize()
            best = max(best, 2.0 * n ** 3 / (e0.elapsed_time(e1) * 1e-3) / 1e12)
        out[name] = best
        del a, b
    torch.backends.cuda.matmul.allow_tf32 = prev
    torch.cuda.empty_cache()
    return out


def j1j2_autompo(tt_b200, Nx, Ny, J2):
    a = tt_b200.AutoMPO()
    for s1, s2, typ, *_ in tt_b200.square_next_neighbor(Nx, Ny, True, snake=True):
        J = 1.0 if typ == 1 else J2
        a.add(0.5 * J, "S+", s1 - 1, "S-", s2 - 1)
        a.add(0.5 * J, "S-", s1 - 1, "S+", s2 - 1)
        a.add(J, "Sz", s1 - 1, "Sz", s2 - 1)
    return a


# ---------------------------------------------------------------------------
# CPU restatement (oracle) on the J1-J2 cylinder at bond dimension 3072
# ---------------------------------------------------------------------------
class OracleMidChain:
    """Real two-site updates of the oracle (update_site + update_env,
    algos/dmrg/dmrg.cpp:300-372,491-509) at bond dimension chi in the middle
    of the 96-site cylinder.  The state is the Neel product state of the
    reference's product-state constructor (mps/qtt.cpp:205-311) with sites
    m-w .. m-1 replaced by random left-canonical and sites m+2 .. m+1+w by
    random right-canonical isometries whose bonds grow to chi (sector
    dimensions binomial, scaled down proportionally once above chi), and a
    random two-site pair at m, m+1; the environments are contracted through
    it with the J1-J2 MPO exactly as buildEnv does, so H_eff is the true
    effective Hamiltonian of that state (Hermitian, identity norm)."""

    def __init__(self, chi, max_restart, cutoff=1e-10, w=12, seed=0):
        import numpy as np
        from oracle import autompo as am, qdmrg
        from oracle.qtensor import QIndex, QTensor, Inward, Outward, Link, qadd
        self.np, self.qdmrg = np, qdmrg
        self.chi, self.max_restart, self.cutoff = chi, max_restart, cutoff
        rng = np.random.default_rng(seed)
        self.rng = rng
        N, m = C5_N, C5_MID
        self.m = m
        a = am.AutoMPO()
        for s1, s2, t, *_ in am.snake_relabel(am.square_next_neighbor(C5["Nx"], C5["Ny"], True), C5["Nx"], C5["Ny"]):
            J = 1.0 if t == 1 else C5["J2"]
            a.add(0.5 * J, "S+", s1 - 1, "S-", s2 - 1)
            a.add(0.5 * J, "S-", s1 - 1, "S+", s2 - 1)
            a.add(J, "Sz", s1 - 1, "Sz", s2 - 1)
        self.H = am.build_qmpo(a, N)
        psi = qdmrg.QMPS(N, qdmrg.neel(N))
        self.psi = psi
        phy = psi.phy_qn
        st = qdmrg.neel(N)
        cum = [(0, 0)]
        for i in range(N):
            cum.append(qadd(cum[-1], phy[st[i]]))

        def cap(d):
            # proportional to the binomial counts, exactly chi in all
            # (largest remainders), empty sectors dropped
            tot = sum(d.values())
            if tot <= chi:
                return dict(d)
            share = {q: v * chi / tot for q, v in d.items()}
            out = {q: int(s) for q, s in share.items()}
            for q in sorted(share, key=lambda q: (out[q] - share[q], q))[:chi - sum(out.values())]:
                out[q] += 1
            return {q: v for q, v in out.items() if v > 0}

        def window(i_from, i_to, step):
            if step > 0:
                prev, active, sites = psi.A[i_from].idx[0].copy(), {cum[i_from]: 1}, range(i_from, i_to)
            else:
                prev, active, sites = psi.A[i_from].idx[2].copy(), {cum[i_from + 1]: 1}, range(i_from, i_to, -1)
            for i in sites:
                nd = {}
                for q, d in active.items():
                    for p in phy:
                        qq = qadd(q, p) if step > 0 else (q[0] - p[0], q[1] - p[1])
                        nd[qq] = nd.get(qq, 0) + d
                nd = cap(nd)
                new = QIndex(Outward, psi.link_name(i + 1), Link, 0) if step > 0 else \
                    QIndex(Inward, psi.link_name(i), Link, 0)
                for q in sorted(nd):
                    new.add_qn(q, nd[q])
                T = QTensor([prev, psi.A[i].idx[1].copy(), new] if step > 0 else [new, psi.A[i].idx[1].copy(), prev])
                T.init_block()
                oa, na = (0, 2) if step > 0 else (2, 0)
                groups = {}
                for b, qi in enumerate(T.bqi):
                    if T.idx[oa].qn(qi[oa]) in active:
                        groups.setdefault(qi[na], []).append(b)
                for bl in groups.values():
                    shapes = [T.blocks[b].shape for b in bl]
                    rows = [s[0] * s[1] if step > 0 else s[1] * s[2] for s in shapes]
                    ncol = shapes[0][2] if step > 0 else shapes[0][0]
                    Q, _ = np.linalg.qr(rng.standard_normal((sum(rows), ncol)))
                    off = 0
                    for b, r, s in zip(bl, rows, shapes):
                        blk = Q[off:off + r]
                        off += r
                        T.blocks[b][...] = (blk if step > 0 else blk.T).reshape(s, order="F")
                psi.A[i] = T
                prev, active = new.dagged(), nd
            return prev, active

        lidx, lact = window(m - w, m, +1)
        ridx, ract = window(m + 1 + w, m + 1, -1)
        md = {}
        for q, d in lact.items():
            for p in phy:
                qq = qadd(q, p)
                if any(qadd(qq, p2) in ract for p2 in phy):
                    md[qq] = md.get(qq, 0) + d
        mid = QIndex(Outward, psi.link_name(m + 1), Link, 0)
        for q, d in sorted(cap(md).items()):
            mid.add_qn(q, d)
        Am = QTensor([lidx, psi.A[m].idx[1].copy(), mid])
        An = QTensor([mid.dagged(), psi.A[m + 1].idx[1].copy(), ridx])
        for T in (Am, An):
            T.init_block()
            for b in T.blocks:
                b[...] = rng.standard_normal(b.shape)
        psi.A[m], psi.A[m + 1] = Am, An
        self.bond_dims = (sum(lact.values()), mid.dim(), sum(ract.values()))
        TL, TR = [None] * N, [None] * N
        TL[0] = qdmrg._boundary(psi.A[0].idx[0], self.H.A[0].idx[0])
        for i in range(m):
            TL[i + 1] = qdmrg.env_step(TL[i], psi.A[i], self.H.A[i])
        TR[N - 1] = qdmrg._boundary(psi.A[N - 1].idx[-1], self.H.A[N - 1].idx[-1])
        for i in range(N - 1, m + 1, -1):
            TR[i - 1] = qdmrg.env_step(TR[i], psi.A[i], self.H.A[i])
        self.TL, self.TR = TL, TR
        self.k = 0

    def update(self):
        """One two-site update: left-to-right at m, then right-to-left at m+1, alternately."""
        from oracle import qsvd
        q = self.qdmrg
        if self.k % 2 == 0:
            e = q.update_site(self.psi, self.H, self.TR, self.TL, self.m, qsvd.MoveFromLeft, self.chi, self.cutoff,
                              3, self.max_restart, self.rng)
            q.update_env(self.psi, self.H, self.TR, self.TL, self.m, qsvd.MoveFromLeft)
        else:
            e = q.update_site(self.psi, self.H, self.TR, self.TL, self.m + 1, qsvd.MoveFromRight, self.chi,
                              self.cutoff, 3, self.max_restart, self.rng)
            q.update_env(self.psi, self.H, self.TR, self.TL, self.m + 1, qsvd.MoveFromRight)
        self.k += 1
        return e


def oracle_updates(chi, max_restart, budget_s, max_updates, warmup=0, seed=0):
    """Set-up (untimed), `warmup` untimed oracle updates, then timed updates
    until `max_updates` or the budget is spent (at least one).  Returns (mean
    seconds per update, updates timed, warm-up updates run, set-up seconds,
    bond dims)."""
    t0 = time.perf_counter()
    om = OracleMidChain(chi, max_restart, seed=seed)
    setup = time.perf_counter() - t0
    t_start = time.perf_counter()
    done_w = 0
    t_w = 0.0
    for _ in range(warmup):
        t1 = time.perf_counter()
        om.update()
        done_w += 1
        t_w = time.perf_counter() - t1
        if time.perf_counter() - t_start + (max_updates + warmup - done_w) * t_w > budget_s:
            break  # keep the budget for the timed updates
    times = []
    while len(times) < max(1, max_updates):
        t1 = time.perf_counter()
        om.update()
        times.append(time.perf_counter() - t1)
        if time.perf_counter() - t_start + statistics.mean(times) > budget_s:
            break
    return statistics.mean(times), len(times), done_w, setup, om.bond_dims


def run_reference(args):
    """The reference arm: one step is one real oracle two-site update at the
    workload's bond dimension (the GPU arm's step is a block of eight), run
    on all host cores; W untimed updates first, then K timed ones, within
    --ref-budget seconds."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    if args.workload == "heisenberg":
        return run_heisenberg_reference(args)
    t_upd, n, n_w, setup, dims = oracle_updates(args.maxdim, args.max_restart, args.ref_budget, args.steps,
                                                warmup=args.warmup)
    value = t_upd * C5_UPDATES_PER_SWEEP
    sample = ("%d real oracle two-site updates (Davidson max %d iters + block SVD + environment update) at bond "
              "dims %s in the middle of the 96-site cylinder, %.1f s each, after %d untimed ones (set-up %.0f s "
              "untimed); a step is one update; s/sweep = s/update x %d updates per sweep" %
              (n, args.max_restart, dims, t_upd, n_w, setup, C5_UPDATES_PER_SWEEP))
    cores = os.cpu_count()
    line = {"metric": METRIC, "value": value, "unit": "s/sweep", "n_gpus": args.gpus, "steps": n,
            "warmup": n_w, "ms_per_step": t_upd * 1e3, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic", "config": c5_config(args),
            "impl": "reference",
            "cpu_baseline": {"value": value, "unit": "s/sweep", "cores": cores, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": "s/sweep", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


# ---------------------------------------------------------------------------
# GPU arm on the J1-J2 cylinder
# ---------------------------------------------------------------------------
def c5_setup(tt_b200, H, args, workdir):
    """Untimed ramp in the chosen form, one sweep at maxdim, checkpoint."""
    from oracle import qdmrg
    tt_b200.set_precision(heff=CHOSEN, env=args.env_prec)
    t0 = time.perf_counter()
    try:
        psi = tt_b200.QMPS(C5_N, qdmrg.neel(C5_N))
        run = tt_b200.QDMRG(psi, H)
        energies = []
        ramp = c5_ramp(args)
        n = len(ramp)
        for k, m in enumerate(ramp):
            energies.append(run.sweep(m, C5["cutoff"], args.max_restart, C5["noise0"] * (1.0 - k / n)))
        energies.append(run.sweep(args.maxdim, C5["cutoff"], args.max_restart, 0.0))
        run.finish()
    finally:
        tt_b200.set_precision()
    ck = os.path.join(workdir, "c5_start")
    psi.save(ck)
    info = {"ramp_seconds": time.perf_counter() - t0, "ramp_energies": energies,
            "start_bond_dims_mid": psi.bond_dims()[C5_MID - 1:C5_MID + args.block + 2]}
    del run, psi
    return ck + ".ttmps", info


def heff_parts_summary(a, b):
    """Per-contraction figures of the products between two heff_parts()
    readings: device ms and algorithmic TFLOP/s of L*x and *R, device ms and
    algorithmic GB/s of the middle contraction."""
    ms = [y - x for x, y in zip(a["ms"], b["ms"])]
    fl = [y - x for x, y in zip(a["flops"], b["flops"])]
    mb = b["mid_bytes"] - a["mid_bytes"]
    out = {"ms": {"L*x": ms[0], "*mid": ms[1], "*R": ms[2]},
           "flops": {"L*x": fl[0], "*mid": fl[1], "*R": fl[2]}, "mid_bytes": mb}
    if ms[0] + ms[2] > 0:
        out["L*x_and_*R_tflops"] = (fl[0] + fl[2]) / ((ms[0] + ms[2]) * 1e-3) / 1e12
    if ms[1] > 0:
        out["mid_gbs"] = mb / (ms[1] * 1e-3) / 1e9
    return out


# <Sz_i Sz_j> pairs in the middle of the cylinder (0-based sites, snake order):
# along the snake, one column over, and two columns over
C5_SZSZ_PAIRS = [(47, 48), (47, 47 + C5["Ny"]), (47, 47 + 2 * C5["Ny"])]


def szsz_mpos(tt_b200):
    out = []
    for i, j in C5_SZSZ_PAIRS:
        a = tt_b200.AutoMPO()
        a.add(1.0, "Sz", i, "Sz", j)
        out.append(tt_b200.QMPO.from_autompo(a, C5_N))
    return out


def c5_arm(prec, ck, H, args, ctx, stream, flush, torch, tt_b200, sampler=None, e2e_steps=0, szsz=None):
    """Load, centre to the block, W warm-up and K timed block steps (CUDA
    events on the library stream, L2 flushed before each), then the FP64
    energy, optional end-to-end steps and a full sweep."""
    env_prec = args.env_prec if prec != "fp64" else "fp64"
    tt_b200.set_precision(heff=prec, env=env_prec)
    res = {"precision": prec, "env_precision": env_prec}
    B, mid = args.block, C5_MID
    cut, mr, md = C5["cutoff"], args.max_restart, args.maxdim
    try:
        psi = tt_b200.QMPS.load(ck)
        run = tt_b200.QDMRG(psi, H)
        run.walk(mid, md, cut, mr)

        def step():
            run.walk(mid + B, md, cut, mr)
            return run.walk(mid, md, cut, mr)

        for _ in range(args.warmup):
            step()
        ctx.sync()
        st0, fb0, l0 = run.stats(), tt_b200.davidson_fallbacks(), ctx.launches()
        pc0 = tt_b200.planning_counters()
        pt0 = tt_b200.plan_timers()
        hp0 = tt_b200.heff_parts()
        er0 = tt_b200.eig_redo_count(ctx)
        s0 = len(run.steps())
        if sampler:
            sampler.start()
        times = []
        # NVTX range "c5_timed_<precision>": lets a profiler's launch list cover the timed steps only
        torch.cuda.nvtx.range_push("c5_timed_" + prec)
        # per step: pool GB reserved, plans built, host seconds, of which waiting on the device
        step_pool, step_plans, step_host, step_wait, step_os = [], [], [], [], []
        try:
            import psutil
            proc = psutil.Process()
            psutil.cpu_percent(None)
            cpu0 = proc.cpu_times()
        except Exception:  # load sampling is diagnostic only
            psutil = None
        for _ in range(args.steps):
            flush.zero_()
            torch.cuda.synchronize()
            pa = tt_b200.planning_counters()["plans"]
            w0 = ctx.wait_stats()[0]
            ru0 = resource.getrusage(resource.RUSAGE_SELF)
            tr0 = ctx.pool_trims()
            al0 = ctx.alloc_stats(reset_max=True)
            cs0 = tt_b200.cache_stats()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            h0 = time.perf_counter()
            e0.record(stream)
            step()
            e1.record(stream)
            step_host.append(time.perf_counter() - h0)
            step_wait.append(ctx.wait_stats()[0] - w0)
            ru1 = resource.getrusage(resource.RUSAGE_SELF)
            step_os.append({"user_s": ru1.ru_utime - ru0.ru_utime, "sys_s": ru1.ru_stime - ru0.ru_stime,
                            "minflt": ru1.ru_minflt - ru0.ru_minflt, "majflt": ru1.ru_majflt - ru0.ru_majflt,
                            "nivcsw": ru1.ru_nivcsw - ru0.ru_nivcsw, "pool_trims": ctx.pool_trims() - tr0})
            al1 = ctx.alloc_stats()
            step_os[-1].update({"alloc_s": al1["alloc_s"] - al0["alloc_s"], "alloc_max_s": al1["alloc_max_s"],
                                "free_s": al1["free_s"] - al0["free_s"], "free_max_s": al1["free_max_s"],
                                "allocs": al1["allocs"] - al0["allocs"],
                                "cache_hits": al1["cache_hits"] - al0["cache_hits"],
                                "cached_gb": al1["cached_bytes"] / 2 ** 30})
            e1.synchronize()
            times.append(e0.elapsed_time(e1) * 1e-3)
            step_plans.append(tt_b200.planning_counters()["plans"] - pa)
            cs1 = tt_b200.cache_stats()
            step_os[-1].update({"cache_entries": cs1["entries"], "cache_plan_gb": cs1["plan_bytes"] / 2 ** 30,
                                "cache_evicted": cs1["evicted"] - cs0["evicted"]})
            step_pool.append(ctx.memory()[2] / 2 ** 30)
        torch.cuda.nvtx.range_pop()
        ctx.sync()
        clocks = sampler.stop() if sampler else None
        st1, launches = run.stats(), ctx.launches() - l0
        pc1 = tt_b200.planning_counters()
        hp1 = tt_b200.heff_parts()
        er1 = tt_b200.eig_redo_count(ctx)
        steps = run.steps()[s0:]
        prof_t = run.profile()[s0:s0 + args.steps * 2 * B]  # host wall time per update, no added syncs
        prof_d = run.device_profile(s0)[:args.steps * 2 * B]  # device-stream spans per update (events)
        t_step = statistics.mean(times)
        upd = 2 * B
        fl = st1["heff_flops"] - st0["heff_flops"]
        hs = st1["heff_seconds"] - st0["heff_seconds"]
        res.update({
            "value": t_step / upd * C5_UPDATES_PER_SWEEP, "unit": "s/sweep", "ms_per_step": t_step * 1e3,
            "step_seconds": times, "s_per_update": t_step / upd,
            "heff_tflops": fl / hs / 1e12 if hs > 0 else 0.0,
            "heff_share_of_step": hs / sum(times) if times else None,
            "heff_tflop_per_step": fl / max(1, args.steps) / 1e12,
            "gpu_launches": int(launches), "launches_per_step": launches / max(1, args.steps),
            "davidson_fallbacks": tt_b200.davidson_fallbacks() - fb0,
            "host_planning_s_per_update": ((pc1["structure_s"] - pc0["structure_s"]) + (pc1["plan_s"] - pc0["plan_s"]))
            / max(1, args.steps * 2 * B),
            "plans_per_update": (pc1["plans"] - pc0["plans"]) / max(1, args.steps * 2 * B),
            "host_structure_s_per_update": (pc1["structure_s"] - pc0["structure_s"]) / max(1, args.steps * 2 * B),
            "planner_stage_s_per_update": [(b - a) / max(1, args.steps * 2 * B) for a, b in zip(pt0, tt_b200.plan_timers())],
            "eig_redos": er1 - er0,
            "heff_parts": heff_parts_summary(hp0, hp1),
            "step_plans_built": step_plans, "step_pool_reserved_gb": step_pool,
            "step_host_seconds": step_host, "step_device_wait_seconds": step_wait, "step_os": step_os,
            # per timed step, host wall seconds inside Davidson (of which building the
            # product engine), the block SVD and the environment update
            "step_host_phases": [
                {"davidson": sum(p[1] for p in prof_t[k * 2 * B:(k + 1) * 2 * B]),
                 "engine": sum(p[4] for p in prof_t[k * 2 * B:(k + 1) * 2 * B]),
                 "svd": sum(p[2] for p in prof_t[k * 2 * B:(k + 1) * 2 * B]),
                 "env": sum(p[3] for p in prof_t[k * 2 * B:(k + 1) * 2 * B])} for k in range(args.steps)],
            # per timed step, device-stream milliseconds of the same phases, and of the
            # gaps between consecutive updates of the step (device waiting for the host)
            "step_device_phases_ms": [
                {"davidson": sum(p[0] for p in prof_d[k * 2 * B:(k + 1) * 2 * B]),
                 "svd": sum(p[1] for p in prof_d[k * 2 * B:(k + 1) * 2 * B]),
                 "env": sum(p[2] for p in prof_d[k * 2 * B:(k + 1) * 2 * B]),
                 "gaps": sum(p[3] for p in prof_d[k * 2 * B + 1:(k + 1) * 2 * B])} for k in range(args.steps)],
            "matvecs_per_update": statistics.mean(s["matvecs"] for s in steps) if steps else None,
            "trunc_err_mean": statistics.mean(s["trunc_err"] for s in steps) if steps else None,
            "kept": [s["kept"] for s in steps[-upd:]],
            "bond_dims_block": psi.bond_dims()[mid:mid + B + 2],
            "clocks": clocks,
        })
        if psutil is not None:
            cpu1 = proc.cpu_times()
            res["host_load"] = {"system_cpu_percent": psutil.cpu_percent(None), "cores": psutil.cpu_count(),
                                "this_process_cpu_s": (cpu1.user + cpu1.system) - (cpu0.user + cpu0.system),
                                "timed_s": sum(times)}
        pool = ctx.memory()
        res["device_memory_gb"] = {"in_use": pool[0] / 2 ** 30, "high_water": pool[1] / 2 ** 30,
                                   "reserved": pool[2] / 2 ** 30}
        if args.breakdown:
            lib = tt_b200.lib
            lib.tt_dmrg_set_profiling(1)
            n0 = len(run.profile())
            try:
                step()
            finally:
                lib.tt_dmrg_set_profiling(0)
            prof = run.profile()[n0:]
            res["breakdown_s_per_update"] = {
                "davidson": statistics.mean(p[1] for p in prof), "svd": statistics.mean(p[2] for p in prof),
                "env": statistics.mean(p[3] for p in prof), "largest_svd_sector": max(p[0] for p in prof)}
        # FP64 energy of the state after the identical schedule
        tt_b200.set_precision()
        nrm = psi.overlap()
        res["energy"] = psi.expectation(H) / nrm
        if szsz:
            res["szsz"] = [psi.expectation(m) / nrm for m in szsz]
        tt_b200.set_precision(heff=prec, env=env_prec)
        if e2e_steps > 0:
            # through the public C ABI: the block's site tensors from pinned host memory every step
            first, last = mid, mid + B + 2
            n_el = psi.sites_size(first, last)
            host = torch.empty(n_el, dtype=torch.float64, pin_memory=True).numpy()
            psi.get_sites(first, last, host)
            e2e, h2d = [], []
            # one untimed step first: the energy and correlator evaluations above
            # ran other contractions through the plan and block caches
            for k in range(1 + e2e_steps):
                ctx.sync()
                t0 = time.perf_counter()
                psi.set_sites(first, last, host)
                step()
                n_el = psi.sites_size(first, last)
                if host.size != n_el:
                    host = torch.empty(n_el, dtype=torch.float64, pin_memory=True).numpy()
                psi.get_sites(first, last, host)
                if k > 0:
                    e2e.append(time.perf_counter() - t0)
                    h2d.append(n_el * 8)
            t = statistics.mean(e2e)
            res["e2e"] = {"value": t / upd * C5_UPDATES_PER_SWEEP, "unit": "s/sweep",
                          "h2d_bytes_per_step": int(statistics.mean(h2d)), "d2h_bytes_per_step": int(statistics.mean(h2d)),
                          "ms_per_step": t * 1e3,
                          "includes": "host->device copy of the block's %d site tensors from pinned memory, the "
                                      "%d-update block step, device->host copy of the updated tensors" % (B + 2, upd)}
        if not args.no_full_sweep:
            try:
                run.walk(0, md, cut, mr)
                ctx.sync()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                e_sweep = run.sweep(md, cut, mr)
                e1.record(stream)
                e1.synchronize()
                res["full_sweep"] = {"seconds": e0.elapsed_time(e1) * 1e-3, "energy": e_sweep,
                                     "max_bond_dim": max(psi.bond_dims())}
            except tt_b200.TTError as exc:  # reported, not fatal: the timed steps stand
                res["full_sweep"] = {"error": str(exc)}
            pool = ctx.memory()
            res["device_memory_gb"]["high_water_with_full_sweep"] = pool[1] / 2 ** 30
        del run, psi
    finally:
        tt_b200.set_precision()
    return res


def _rounded(x):
    if isinstance(x, dict):
        return {k: _rounded(v) for k, v in x.items()}
    if isinstance(x, (list, tuple)):
        return [_rounded(v) for v in x]
    return float("%.7g" % x) if isinstance(x, float) else x


def compact(out):
    """The result line of what --detail writes: without the texts that explain a number, of the two arms what their
    comparison needs, numbers with seven digits (energies in full)."""
    line = {k: _rounded(v) for k, v in out.items() if k not in ("mixed", "fp64")}
    for name, keys in (("config", ("ramp_seconds", "ramp_energies", "start_bond_dims_mid", "setup", "value_definition")),
                       ("roofline", ("peak_source", "tf32_products_frac")), ("e2e", ("includes",)),
                       ("cpu_baseline", ("sample",))):
        for k in keys:
            (line.get(name) or {}).pop(k, None)
    short = ("value", "ms_per_step", "heff_share_of_step", "heff_tflops", "launches_per_step", "speedup_vs_fp64")
    full = ("energy", "dE_per_site_vs_fp64", "szsz_max_abs_err_vs_fp64", "full_sweep")
    for name in ("mixed", "fp64"):
        arm = out[name]
        line[name] = {k: _rounded(arm[k]) for k in short if k in arm}
        line[name].update({k: arm[k] for k in full if k in arm})
        if "step_seconds" in arm:
            line[name]["step_seconds_min_max"] = _rounded([min(arm["step_seconds"]), max(arm["step_seconds"])])
        line[name]["kernel_fracs"] = {k: _rounded(r["frac"]) for k, r in arm.get("kernel_rooflines", {}).items()}
    return line


def run_c5(args):
    import torch
    import tt_b200

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=900))

    def barrier():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()

    peaks = measured_peaks(torch)
    ctx = tt_b200.Context(local)
    stream = torch.cuda.ExternalStream(ctx.stream())
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    H = tt_b200.QMPO.from_autompo(j1j2_autompo(tt_b200, C5["Nx"], C5["Ny"], C5["J2"]), C5_N)
    workdir = tempfile.mkdtemp(prefix="tt_c5_")
    try:
        ck, setup = c5_setup(tt_b200, H, args, workdir)
        barrier()
        sampler = None if args.no_clock_sampler else ClockSampler(local)
        sz = szsz_mpos(tt_b200)
        chosen = c5_arm(CHOSEN, ck, H, args, ctx, stream, flush, torch, tt_b200, sampler=sampler,
                        e2e_steps=args.e2e_steps, szsz=sz)
        print("[bench] %s arm: %.3f s/sweep, pool GB %s" % (CHOSEN, chosen["value"], ["%.1f" % (v / 2 ** 30)
                                                             for v in ctx.memory()]), file=sys.stderr, flush=True)
        barrier()
        fp64 = c5_arm("fp64", ck, H, args, ctx, stream, flush, torch, tt_b200, szsz=sz)
        barrier()
    finally:
        shutil.rmtree(workdir, ignore_errors=True)
    # replicas: every rank runs its own copy of the problem (the path does not
    # shard); the reported time is the slowest rank's, per GPU
    t_max = chosen["value"]
    if dist is not None:
        t = torch.tensor([t_max], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        t_max = float(t.item())
    out = None
    if rank == 0:
        cpu = None
        if not args.no_cpu_baseline:
            t_upd, n, _, setup_s, dims = oracle_updates(args.maxdim, args.max_restart, args.cpu_budget, 1)
            cpu = {"value": t_upd * C5_UPDATES_PER_SWEEP, "unit": "s/sweep", "cores": os.cpu_count(),
                   "kind": "port",
                   "sample": "%d real oracle two-site update(s) at bond dims %s in the middle of the cylinder "
                             "(%.1f s each; set-up %.0f s untimed) x %d updates per sweep" % (
                                 n, dims, t_upd, setup_s, C5_UPDATES_PER_SWEEP)}
        de = abs(chosen["energy"] - fp64["energy"]) / C5_N
        chosen["dE_per_site_vs_fp64"] = de
        if "szsz" in chosen and "szsz" in fp64:
            chosen["szsz_pairs"] = C5_SZSZ_PAIRS
            chosen["szsz_max_abs_err_vs_fp64"] = max(abs(a - b) for a, b in zip(chosen["szsz"], fp64["szsz"]))
        chosen["speedup_vs_fp64"] = fp64["value"] / chosen["value"]
        if "seconds" in chosen.get("full_sweep", {}) and "seconds" in fp64.get("full_sweep", {}):
            chosen["full_sweep"]["speedup_vs_fp64"] = fp64["full_sweep"]["seconds"] / chosen["full_sweep"]["seconds"]
            chosen["full_sweep"]["dE_per_site_vs_fp64"] = abs(chosen["full_sweep"]["energy"] -
                                                              fp64["full_sweep"]["energy"]) / C5_N
        chosen["roofline"] = {
            "bound": "tensor", "kernel": "H_eff*x: grouped_tc_persist (3xTF32 tcgen05) for L*x and *R, "
                                         "narrow_dgemm (FP64) for the middle contraction",
            "achieved": chosen["heff_tflops"], "peak": peaks["tf32"] / 3.0, "unit": "TFLOP/s",
            "frac": chosen["heff_tflops"] / (peaks["tf32"] / 3.0),
            "peak_source": "cuBLAS TF32 GEMM 8192^3 measured in this run (%.1f TFLOP/s) / 3: each algorithmic "
                           "3xTF32 flop is three TF32 products" % peaks["tf32"],
            "tf32_products_frac": 3.0 * chosen["heff_tflops"] / peaks["tf32"], "traffic": None}
        hbm = load_hbm_peak()
        for arm, peak_tc, kind in ((chosen, peaks["tf32"] / 3.0, "3xTF32 tcgen05 (grouped_tc_persist)"),
                                   (fp64, peaks["fp64"], "FP64 DMMA (grouped_dgemm)")):
            hpts = arm.get("heff_parts", {})
            kr = {}
            if "L*x_and_*R_tflops" in hpts:
                kr["L*x and *R"] = {"bound": "tensor", "kernel": kind, "achieved": hpts["L*x_and_*R_tflops"],
                                    "peak": peak_tc, "unit": "TFLOP/s",
                                    "frac": hpts["L*x_and_*R_tflops"] / peak_tc}
            if "mid_gbs" in hpts and hbm:
                kr["*mid"] = {"bound": "hbm", "kernel": "narrow_dgemm (FP64)", "achieved": hpts["mid_gbs"],
                              "peak": hbm, "unit": "GB/s", "frac": hpts["mid_gbs"] / hbm,
                              "peak_source": "MEASURED_PEAKS.json hbm_gbs (copy bandwidth)"}
            arm["kernel_rooflines"] = kr
        fp64["roofline"] = {
            "bound": "tensor", "kernel": "H_eff*x: grouped_dgemm (DMMA), 3 launches per product",
            "achieved": fp64["heff_tflops"], "peak": peaks["fp64"], "unit": "TFLOP/s",
            "frac": fp64["heff_tflops"] / peaks["fp64"],
            "peak_source": "cuBLAS DGEMM 8192^3 measured in this run", "traffic": None}
        out = {
            "metric": METRIC, "value": t_max, "unit": "s/sweep", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": chosen["ms_per_step"], "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None, "dtype": "tf32x3+f64", "data": "synthetic",
            "config": dict(c5_config(args), precision=CHOSEN + ": 3xTF32 tcgen05 or FP64 DMMA per contraction "
                           "(cost model) for H_eff*x; FP64 environments, Gram-Schmidt, Rayleigh-Ritz, block "
                           "SVD and energies", parallelism="replicas" if world > 1 else "single", **setup),
            "heff_tflops": chosen["heff_tflops"],
            "roofline": chosen["roofline"],
            "cpu_baseline": cpu,
            "e2e": chosen.get("e2e"),
            "gpu_launches": chosen["gpu_launches"],
            "clocks": chosen["clocks"],
            "mixed": chosen,
            "fp64": fp64,
            "peaks_measured": peaks,
        }
        if args.detail:
            with open(args.detail, "w") as f:
                json.dump(out, f)
        print(json.dumps(compact(out)))
    ctx.close()
    if dist is not None:
        dist.destroy_process_group()


# ---------------------------------------------------------------------------
# secondary workload: Heisenberg chain L = 100 to maxdim 512
# ---------------------------------------------------------------------------
HEIS = dict(L=100, ramp=(32, 64, 128, 256), maxdim=512, cutoff=1e-12, max_restart=6)


def heis_config():
    return {"workload": "U(1) two-site DMRG, spin-1/2 Heisenberg chain J=1 OBC L=100, Sz=0 Neel start, maxdim 512 "
                        "(after untimed ramp 32,64,128,256), cutoff 1e-12, Davidson max 6 iters (tol 1e-12 as "
                        "hard-wired in the reference; the configuration's 1e-11 is looser)",
            "L": HEIS["L"], "maxdim": HEIS["maxdim"], "cutoff": HEIS["cutoff"], "max_restart": HEIS["max_restart"],
            "step": "one full sweep (L->R + R->L, 2x99 two-site updates)",
            "l2": "L2 flushed before each timed sweep"}


def oracle_heisenberg_sweeps(budget_s):
    """The oracle's own schedule: untimed ramp 32..256, then timed full sweeps
    at maxdim 512 until the budget is spent (at least one)."""
    from oracle import qdmrg
    L = HEIS["L"]
    psi = qdmrg.QMPS(L, qdmrg.neel(L))
    H = qdmrg.QMPO(L)
    t0 = time.perf_counter()
    qdmrg.dmrg(psi, H, len(HEIS["ramp"]), list(HEIS["ramp"]), [HEIS["cutoff"]], [HEIS["max_restart"]])
    setup = time.perf_counter() - t0
    times = []
    while True:
        t1 = time.perf_counter()
        qdmrg.dmrg(psi, H, 1, [HEIS["maxdim"]], [HEIS["cutoff"]], [HEIS["max_restart"]])
        times.append(time.perf_counter() - t1)
        if sum(times) + statistics.mean(times) > budget_s:
            break
    return statistics.mean(times), len(times), setup


def run_heisenberg_reference(args):
    t, n, setup = oracle_heisenberg_sweeps(args.ref_budget)
    print(json.dumps({"metric": METRIC, "value": t, "unit": "s/sweep", "n_gpus": args.gpus, "steps": n,
                      "warmup": 0, "ms_per_step": t * 1e3, "higher_is_better": False, "scaling": "weak",
                      "vs_baseline": None, "dtype": "f64", "data": "synthetic", "config": heis_config(),
                      "impl": "reference",
                      "cpu_baseline": {"value": t, "unit": "s/sweep", "cores": os.cpu_count(), "kind": "port",
                                       "sample": "%d full oracle sweeps at maxdim 512 after its own ramp (%.0f s "
                                                 "untimed)" % (n, setup)},
                      "e2e": {"value": t, "unit": "s/sweep", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}))


def run_heisenberg(args):
    import torch
    import tt_b200
    from oracle import qdmrg
    L = HEIS["L"]
    ctx = tt_b200.Context(0)
    stream = torch.cuda.ExternalStream(ctx.stream())
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    peaks = measured_peaks(torch)
    out = {}
    for prec in ("fp64", CHOSEN):
        tt_b200.set_precision(heff=prec, env=prec)
        try:
            psi = tt_b200.QMPS(L, qdmrg.neel(L))
            H = tt_b200.QMPO(L)
            run = tt_b200.QDMRG(psi, H)
            for m in HEIS["ramp"]:
                run.sweep(m, HEIS["cutoff"], HEIS["max_restart"])
            for _ in range(args.warmup):
                run.sweep(HEIS["maxdim"], HEIS["cutoff"], HEIS["max_restart"])
            st0, l0 = run.stats(), ctx.launches()
            ms, energy = [], None
            for _ in range(args.steps):
                flush.zero_()
                torch.cuda.synchronize()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                energy = run.sweep(HEIS["maxdim"], HEIS["cutoff"], HEIS["max_restart"])
                e1.record(stream)
                e1.synchronize()
                ms.append(e0.elapsed_time(e1))
            st1 = run.stats()
            fl, hs = st1["heff_flops"] - st0["heff_flops"], st1["heff_seconds"] - st0["heff_seconds"]
            out[prec] = {"value": statistics.mean(ms) * 1e-3, "unit": "s/sweep", "energy": energy,
                         "heff_tflops": fl / hs / 1e12 if hs else 0.0, "launches_per_sweep":
                             (ctx.launches() - l0) / max(1, args.steps), "bond_dims_mid": psi.bond_dims()[L // 2]}
            del run, psi, H
        finally:
            tt_b200.set_precision()
    ctx.close()
    f = out["fp64"]
    cpu = None
    if not args.no_cpu_baseline:
        t, n, setup = oracle_heisenberg_sweeps(args.cpu_budget)
        cpu = {"value": t, "unit": "s/sweep", "cores": os.cpu_count(), "kind": "port",
               "sample": "%d full oracle sweeps at maxdim 512 after its own ramp (%.0f s untimed)" % (n, setup)}
    out[CHOSEN]["dE_per_site_vs_fp64"] = abs(out[CHOSEN]["energy"] - f["energy"]) / L
    print(json.dumps({"metric": METRIC, "value": f["value"], "unit": "s/sweep", "n_gpus": 1, "steps": args.steps,
                      "warmup": args.warmup, "ms_per_step": f["value"] * 1e3, "higher_is_better": False,
                      "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
                      "config": dict(heis_config(), precision="FP64 (plain GPU form)"),
                      "heff_tflops": f["heff_tflops"],
                      "roofline": {"bound": "tensor", "kernel": "grouped_dgemm", "achieved": f["heff_tflops"],
                                   "peak": peaks["fp64"], "unit": "TFLOP/s", "frac": f["heff_tflops"] / peaks["fp64"],
                                   "peak_source": "cuBLAS DGEMM 8192^3 measured in this run", "traffic": None},
                      "cpu_baseline": cpu, "mixed": out[CHOSEN], "peaks_measured": peaks}))


# ---------------------------------------------------------------------------
def run_chains(args):
    """Independent XXZ chains with site fields (the batched-chains configuration:
    L ~ U{32..128}, Delta ~ U[0.5, 1.5], h_i ~ U[-0.1, 0.1], seed 7, Sz=0 Neel
    start, maxdim ramp 32, 64, 128, 256), solved one after another on one
    context and then concurrently on `--streams` contexts (one host thread and
    CUDA stream each); wall time over the whole batch."""
    import numpy as np
    import tt_b200
    from tt_b200 import replicas
    from oracle import qdmrg
    rng = np.random.default_rng(7)
    items = [(int(L), float(d), list(rng.uniform(-0.1, 0.1, int(L))))
             for L, d in zip(rng.integers(32, 129, args.chains), rng.uniform(0.5, 1.5, args.chains))]
    sched = [32, 64, 128, 256][:max(1, args.chain_sweeps)] + [256] * max(0, args.chain_sweeps - 4)

    def solve(item):
        L, delta, h = item
        a = tt_b200.AutoMPO()
        for i in range(L - 1):
            a.add(0.5, "S+", i, "S-", i + 1).add(0.5, "S-", i, "S+", i + 1).add(delta, "Sz", i, "Sz", i + 1)
        for i in range(L):
            a.add(h[i], "Sz", i)
        psi = tt_b200.QMPS(L, qdmrg.neel(L))
        run = tt_b200.QDMRG(psi, tt_b200.QMPO.from_autompo(a, L))
        e = run.run(len(sched), sched, [1e-10], [6])
        del run, psi
        return e

    t0 = time.perf_counter()
    ctx = tt_b200.Context(0)
    seq = [solve(it) for it in items]
    ctx.close()
    t_seq = time.perf_counter() - t0
    t0 = time.perf_counter()
    conc = replicas.run_chains_concurrent(items, solve, streams=args.streams)
    t_conc = time.perf_counter() - t0
    sweeps = len(items) * len(sched)
    print(json.dumps({
        "metric": "independent chains: chain-sweeps per second (one GPU)", "value": sweeps / t_conc,
        "unit": "chain-sweeps/s", "n_gpus": 1, "higher_is_better": True, "dtype": "f64", "data": "synthetic",
        "config": {"workload": "%d XXZ chains with fields, L in [32,128], maxdim %s" % (len(items), sched),
                   "streams": args.streams},
        "sequential": {"value": sweeps / t_seq, "unit": "chain-sweeps/s", "seconds": t_seq},
        "concurrent_seconds": t_conc, "speedup": t_seq / t_conc,
        "max_energy_difference": max(abs(a - b) for a, b in zip(seq, conc))}))


def run_gemm(args):
    """Throughput of the grouped contraction kernels on one large block: C(m, n)
    = A(m, k) B(k, n), m = n = k = --gemm-size, random FP64 operands, as a
    qtensor contraction with one sector per index; W untimed and K timed
    launches per precision, CUDA events on the library stream.  The
    mixed-precision times include the packing of both operands."""
    import numpy as np
    import torch
    import tt_b200
    from oracle.qtensor import QIndex, QTensor, Inward, Outward, Link, qn
    ctx = tt_b200.Context(0)
    stream = torch.cuda.ExternalStream(ctx.stream())
    n = args.gemm_size
    rng = np.random.default_rng(0)

    def idx(arrow, name):
        ix = QIndex(arrow, name, Link, 0)
        ix.add_qn(qn(0), n)
        return ix

    i, k, j = idx(Inward, "i"), idx(Outward, "k"), idx(Inward, "j")
    A = QTensor([i, k])
    A.init_block()
    A.blocks[0][...] = rng.standard_normal((n, n))
    B = QTensor([k.dagged(), j])
    B.init_block()
    B.blocks[0][...] = rng.standard_normal((n, n))
    gA, gB = tt_b200.QTensor.from_oracle(A), tt_b200.QTensor.from_oracle(B)
    out = {}
    for prec in args.precisions.split(","):
        tt_b200.set_precision(op=prec)
        for _ in range(args.warmup):
            C = gA * gB
        ctx.sync()
        ms = 0.0
        for _ in range(args.steps):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            C = gA * gB
            e1.record(stream)
            e1.synchronize()
            ms += e0.elapsed_time(e1)
            del C
        out[prec] = {"ms": ms / args.steps, "tflops": 2.0 * n ** 3 / (ms / args.steps * 1e-3) / 1e12}
    tt_b200.set_precision()
    print(json.dumps({"metric": "single-block contraction throughput", "unit": "TFLOP/s (algorithmic)",
                      "config": {"workload": "C = A B, %d^3, one QN sector" % n, "steps": args.steps,
                                 "warmup": args.warmup}, "results": out}))
    del gA, gB
    ctx.close()


def main():
    args = parse()
    if args.impl == "reference":
        if args.workload in ("j1j2", "heisenberg"):
            run_reference(args)
        else:
            print(json.dumps({"impl": "reference", "unavailable": "the reference arm covers the j1j2 and "
                                                                  "heisenberg workloads"}))
    elif args.workload == "xxz-chains":
        run_chains(args)
    elif args.workload == "gemm":
        run_gemm(args)
    elif args.workload == "heisenberg":
        run_heisenberg(args)
    else:
        run_c5(args)


if __name__ == "__main__":
    main()
