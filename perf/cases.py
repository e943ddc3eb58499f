"""The calls a user of this engine makes, as measurable cases.

Each case is one pass through a public entry point: the batched FP32 overlap
energy (device-resident and host buffers), the FP64 energy recompute, the FP64
polish, the interval certifier (one packing and a batch), the annealer (one
job, a batch of jobs, the reference-style target-ladder search) and the
continuous-batching server.  ``listed`` names twelve of them from the smallest
call to the largest; ``draw`` gives others of the same ranges.
"""
from __future__ import annotations

import ctypes as C
import math
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "squares-in-squares_b200"))

from sqs import Context, core, polish, sat  # noqa: E402
from sqs import _native as N  # noqa: E402
from sqs.anneal import AnnealJob, _cjob, anneal_batch, jittered_grid, portfolio  # noqa: E402
from sqs.serve import Server  # noqa: E402
from sqs.workloads import certify_corpus, sat_microbench  # noqa: E402


def listed():
    return [
        # a handful of small configurations on the device: what an interactive
        # search evaluates per step, bound by the launch
        dict(name="energy: 48 x n=17", kind="energy", configs=48, n=17, count=False),
        # the benchmark's batch: 4,096 random configurations of 200 squares
        dict(name="energy: 4096 x n=200", kind="energy", configs=4096, n=200, count=False),
        # the largest states the engine takes, candidate pairs counted
        dict(name="energy: 1500 x n=999", kind="energy", configs=1500, n=999, count=True),
        # the same energy called on host arrays, a ragged batch
        dict(name="energy from host: 777 x n=333", kind="energy_host", configs=777, n=333, count=True),
        # FP64 recompute of a search's candidate states, every size of the competition
        dict(name="energy FP64 400 of n 5-1000", kind="energy_fp64", count=400, n_lo=5, n_hi=1000),
        # polish of a campaign's raw states, half of them overlapped
        dict(name="polish: 64 of n 5-1000", kind="polish", count=64, n_lo=5, n_hi=1000, iters=200),
        # the gate on one candidate packing, as each merge step calls it
        dict(name="certify: 1 of n 40-60", kind="certify", count=1, n_lo=40, n_hi=60, roundtrip=False),
        # validation of a batch of submissions: exact grids, near-contact lattices, injected overlaps
        dict(name="certify: 1500 of n 5-1000", kind="certify", count=1500, n_lo=5, n_hi=1000, roundtrip=False),
        # the plain single-instance job: n = 10, 8 replicas, polish and certificate
        dict(name="anneal: n=10 x 8 replicas", kind="anneal", n=10, replicas=8, sweeps=4000),
        # one batched launch of many instances: n uniform in [20, 400], 32 replicas
        dict(name="anneal batch: 256 x 32", kind="anneal_batch", count=256, n_lo=20, n_hi=400, replicas=32, sweeps=50),
        # the drop-in search programs' call: ladders of 8 chains below a shared best side
        dict(name="search: n=50: 64 chains", kind="search", n=50, ladders=8, epochs=40, steps=64),
        # a burst of served jobs of mixed sizes
        dict(name="serve: 32 jobs of n 5-300", kind="serve", count=32, n_lo=5, n_hi=300, sweeps=200),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "energy", "energy_host", "energy_fp64", "polish", "certify", "certify", "anneal",
                       "anneal_batch", "search", "serve"])
    if kind in ("energy", "energy_host"):
        n = _log_int(rng, 2, 1000)
        configs = _log_int(rng, 1, max(2, min(8192, (1_500_000 if kind == "energy" else 400_000) // n)))
        return dict(kind=kind, configs=configs, n=n, count=rng.random() < 0.5)
    hi = _log_int(rng, 12, 1000)
    if kind == "energy_fp64":
        return dict(kind=kind, count=_log_int(rng, 1, 400), n_lo=5, n_hi=hi)
    if kind == "polish":
        return dict(kind=kind, count=_log_int(rng, 1, 64), n_lo=5, n_hi=hi, iters=rng.choice([50, 100, 200]))
    if kind == "certify":
        return dict(kind=kind, count=_log_int(rng, 1, 1500), n_lo=5, n_hi=hi, roundtrip=rng.random() < 0.25)
    if kind == "anneal":
        n = _log_int(rng, 5, 400)
        return dict(kind=kind, n=n, replicas=rng.choice([8, 16, 32, 64]), sweeps=max(10, _log_int(rng, 2000, 40_000) // n))
    if kind == "anneal_batch":
        return dict(kind=kind, count=_log_int(rng, 8, 256), n_lo=20, n_hi=_log_int(rng, 40, 400),
                    replicas=rng.choice([8, 16, 32]), sweeps=_log_int(rng, 10, 50))
    if kind == "search":
        return dict(kind=kind, n=_log_int(rng, 5, 100), ladders=rng.choice([1, 2, 4, 8]), epochs=_log_int(rng, 5, 40),
                    steps=rng.choice([32, 48, 64]))
    return dict(kind=kind, count=_log_int(rng, 4, 32), n_lo=5, n_hi=min(hi, 300), sweeps=_log_int(rng, 20, 200))


# ----------------------------------------------------------------- inputs
_KEPT: dict[str, object] = {}


def _ctx() -> Context:
    """The program's context: one for all its calls."""
    if "ctx" not in _KEPT:
        _KEPT["ctx"] = Context(0)
    return _KEPT["ctx"]


def _server() -> Server:
    """The program's server: created once, jobs come and go."""
    if "server" not in _KEPT:
        _KEPT["server"] = Server(_ctx(), hbm_bytes=1 << 30, max_active=64, slice_proposals=4000)
    return _KEPT["server"]


def _buf(t: torch.Tensor):
    """A device buffer as sat.energy_device takes it."""
    return SimpleNamespace(ptr=t.data_ptr())


def _sizes(case):
    """Sizes log-uniform in the case's range, the same for every seed (outputs
    keep their shapes)."""
    rng = np.random.default_rng(7)
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    return [int(round(math.exp(rng.uniform(lo, hi)))) for _ in range(case["count"])]


def _states(case, seed, rough_every=2):
    """Raw states a search hands on: grids a little apart with small jitter
    (a dilation below 1.008 certifies them), every `rough_every`-th one
    overlapped as an unfinished replica is."""
    rng = np.random.default_rng(seed)
    states, sides = [], []
    for k, n in enumerate(_sizes(case)):
        w = math.isqrt(n - 1) + 1
        i = np.arange(n)
        xy = np.stack([i % w + 0.5, i // w + 0.5], axis=1)
        rough = k % rough_every == rough_every - 1
        pitch, jit, ang = (1.0, 0.05, 0.1) if rough else (1.004, 1e-3, 2e-3)
        xy = xy * pitch + rng.uniform(-jit, jit, (n, 2))
        states.append(np.concatenate([xy, rng.uniform(0.0, ang, (n, 1))], axis=1))
        sides.append(w * pitch)
    return states, np.array(sides)


def _call_arrays(jobs):
    """The C ABI's arrays of a batch of jobs."""
    arr = (N.Job * len(jobs))(*[_cjob(j) for j in jobs])
    res = (N.JobResult * len(jobs))()
    outs = [np.zeros((j.n, 3)) for j in jobs]
    ptrs = (C.POINTER(C.c_double) * len(jobs))(*[o.ctypes.data_as(C.POINTER(C.c_double)) for o in outs])
    return SimpleNamespace(jobs=jobs, arr=arr, res=res, outs=outs, ptrs=ptrs)


def _batch_jobs(case, seed):
    jobs = []
    sizes = np.random.default_rng(42).integers(case["n_lo"], case["n_hi"] + 1, case["count"])
    for k, n in enumerate(sizes):
        xya, side = jittered_grid(int(n), seed=seed * 1000 + k)
        jobs.append(AnnealJob(xya, L0=side, replicas=case["replicas"], sweeps=case["sweeps"], exchange_every=10,
                              tmin=1e-4, tmax=5e-2, sigma_xy=0.02, sigma_a=0.05, seed=seed + k, polish_iters=0))
    return jobs


def _search_job(case, seed):
    """bin/seeded's job: every ladder of 8 chains a ladder of rungs below the
    shared best side, a checkpoint after every epoch of `steps` proposals."""
    n, lad = case["n"], case["ladders"]
    xya, side = jittered_grid(n, seed=seed)
    starts = portfolio(xya, side, 8 * lad, seed=seed)
    return AnnealJob(xya, L0=side, replicas=8 * lad, sweeps=-case["epochs"] * case["steps"],
                     exchange_every=-case["steps"], tmin=1e-11, tmax=1e-4, sigma_xy=0.02, sigma_a=0.014,
                     shrink=0.001 / side, seed=seed, polish_iters=120, adapt=True, collective=True, kick=True,
                     quench_all=True, cert_all=True, quench_steps=8, targets=True, ladders=lad,
                     cluster=min(16, 8 * lad), xya_rep=starts)


def _serve_jobs(case, seed):
    rng = np.random.default_rng(seed)
    jobs = []
    for k, n in enumerate(_sizes(case)):
        xya, side = jittered_grid(n, seed=seed * 1000 + k)
        jobs.append(AnnealJob(xya, L0=side, replicas=int(rng.choice([16, 32, 64])), sweeps=case["sweeps"],
                              exchange_every=10, tmin=1e-3, tmax=1e-1, seed=seed + k))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    s = SimpleNamespace(kind=kind, case=case, ctx=_ctx())
    if kind in ("energy", "energy_host"):
        xya, side = sat_microbench(case["configs"], case["n"], seed)
        xya, side = xya.astype(np.float32), side.astype(np.float32)
        if kind == "energy_host":
            s.xya, s.side = xya, side
            return s
        s.xya, s.side = torch.from_numpy(xya).cuda(), torch.from_numpy(side).cuda()
        s.energy = torch.empty(case["configs"], device="cuda")
        s.grad = torch.empty_like(s.xya)
        s.cand = torch.empty(case["configs"], dtype=torch.int32, device="cuda") if case["count"] else None
        s.bufs = [_buf(t) if t is not None else None for t in (s.xya, s.side, s.energy, s.grad, s.cand)]
        s.out = dict(energy=s.energy, grad=s.grad, **({"cand": s.cand} if case["count"] else {}))
        torch.cuda.synchronize()
    elif kind in ("energy_fp64", "polish"):
        s.states, s.sides = _states(case, seed)
    elif kind == "certify":
        s.arrays = core.pack_batch(certify_corpus(case["count"], seed=seed, n_lo=case["n_lo"], n_hi=case["n_hi"]))
    elif kind == "anneal":
        xya, side = jittered_grid(case["n"], seed=seed)
        s.jobs = [AnnealJob(xya, L0=side, replicas=case["replicas"], sweeps=case["sweeps"], exchange_every=10,
                            tmin=1e-3, tmax=1e-1, seed=seed)]
    elif kind == "anneal_batch":
        s.call = _call_arrays(_batch_jobs(case, seed))
    elif kind == "search":
        s.call = _call_arrays([_search_job(case, seed)])
    else:
        s.server, s.jobs = _server(), _serve_jobs(case, seed)
    return s


# ------------------------------------------------------------------ passes
def _text(raw, field):
    """A char field of an array of C structures, as bytes."""
    b = np.frombuffer(raw, np.uint8).reshape(len(raw), C.sizeof(raw) // len(raw))
    return b[:, field.offset:field.offset + field.size]


def _fields(raw, names):
    rec = np.ctypeslib.as_array(raw)
    return {k: rec[k] for k in names}


def _job_outputs(r):
    """One result dictionary of the Python API, without its clock."""
    return dict(q=np.array(r["q"] if r["q"] is not None else np.zeros((r["n"], 3))),
                sides=np.array([r["L_cert"], r["L_polished"], r["dilation"], r["score"]]),
                L=np.frombuffer((r["L"] or "").encode().ljust(80, b"\0"), np.uint8),
                counts=np.array([r["status"], r["certified"], r["shrinks"], r["sweeps"], r["proposals"],
                                 r["accepted"], r["exchange_attempts"], r["exchange_accepts"]], np.int64))


def run(s):
    kind = s.kind
    if kind == "energy":
        sat.energy_device(s.ctx, s.case["configs"], s.case["n"], *s.bufs)
        return s.out
    if kind == "energy_host":
        e, g, c = sat.energy(s.xya, s.side, ctx=s.ctx, grad=True, count=s.case["count"])
        return dict(energy=e, grad=g, **({"cand": c.view(np.int32)} if s.case["count"] else {}))
    if kind == "energy_fp64":
        e, g = sat.energy_fp64(s.states, s.sides, ctx=s.ctx)
        return dict(energy=e, grad=np.concatenate(g))
    if kind == "polish":
        got = polish.polish_batch(s.states, s.case["iters"], ctx=s.ctx)
        return dict(xya=np.concatenate([q for q, _ in got]),
                    sides=np.array([(r["L_in"], r["L_out"]) for _, r in got]),
                    iterations=np.array([r["iterations"] for _, r in got]))
    if kind == "certify":
        v = core.certify_arrays(*s.arrays, roundtrip=s.case["roundtrip"], ctx=s.ctx)
        return dict(_fields(v, ("ok", "n", "score")), L=_text(v, N.Verdict.L), reason=_text(v, N.Verdict.reason))
    if kind == "anneal":
        return _job_outputs(anneal_batch(s.jobs, ctx=s.ctx)[0])
    if kind in ("anneal_batch", "search"):
        c = s.call
        N.check(N.lib().sqs_anneal_batch(s.ctx.handle, c.arr, len(c.jobs), 0, c.ptrs, c.res))
        return dict(_fields(c.res, ("status", "certified", "shrinks", "improvements", "sweeps_done", "overflows",
                                    "L_cert", "L_polished", "dilation", "score", "proposals", "accepted",
                                    "exchange_attempts", "exchange_accepts")),
                    L=_text(c.res, N.JobResult.L), q=np.concatenate(c.outs))
    ids = [s.server.submit(j) for j in s.jobs]
    got = {}
    while len(got) < len(ids):
        s.server.step()
        for jid in ids:
            if jid not in got:
                r = s.server.poll(jid)
                if r is not None:
                    got[jid] = r
    outs = [_job_outputs(got[jid]) for jid in ids]
    return {k: np.concatenate([o[k].reshape(-1) for o in outs]) for k in outs[0]}


# -------------------------------------------------------------------- work
def _mean_n(case):
    """Mean size of a log-uniform draw."""
    lo, hi = case["n_lo"], case["n_hi"]
    return (hi - lo) / math.log(hi / lo) if hi > lo else float(lo)


def work(case):
    kind = case["kind"]
    if kind in ("energy", "energy_host"):
        rows = case["configs"] * case["n"]
        # 24 B a square in and out; about 2.6 pairs a square inside the
        # cut-off at 55 flop, 60 flop of trig and walls
        return dict(bytes=24 * rows + (12 if case["count"] else 8) * case["configs"], flops=rows * (2.6 * 55 + 60))
    if kind == "energy_fp64":
        rows = case["count"] * _mean_n(case)
        return dict(bytes=48 * rows + 16 * case["count"], flops=rows * (4 * 60 + 80))
    if kind == "polish":
        rows = case["count"] * _mean_n(case)
        # each step: a gradient and at least one trial over about 4 partners
        return dict(bytes=48 * rows, flops=rows * case["iters"] * 2 * (4 * 60 + 80))
    if kind == "certify":
        rows = case["count"] * _mean_n(case)
        # about 45 B of literals a row, about 4 close pairs a square at 110 flop
        return dict(bytes=rows * (45 + 24 + 4) + 208 * case["count"], flops=rows * 4 * 110)
    # one proposal: the pair energy before and after against about 4 neighbours
    per = 2 * 4 * 35 + 2 * 10
    if kind == "anneal":
        props = case["n"] * case["sweeps"] * case["replicas"]
        return dict(bytes=48 * case["n"], flops=props * per)
    if kind == "anneal_batch":
        rows = case["count"] * (case["n_lo"] + case["n_hi"]) / 2
        return dict(bytes=48 * rows, flops=rows * case["sweeps"] * case["replicas"] * per)
    if kind == "search":
        chains = 8 * case["ladders"]
        # proposals, and at every epoch a quench of up to 128 steps of two evaluations
        quench = case["epochs"] * 128 * case["n"] * 2 * (4 * 55 + 60)
        return dict(bytes=24 * case["n"] * (chains + 1),
                    flops=chains * (case["epochs"] * case["steps"] * per + quench))
    rows = case["count"] * _mean_n(case)
    return dict(bytes=48 * rows, flops=rows * case["sweeps"] * 37 * per)


# ------------------------------------------------------------------- exact
def _exact_energy(xya, side, grad_of=True):
    """Walls + squared SAT penetration of every pair and the gradient, in 64
    bits: xya (configs, n, 3), side (configs,) float64 tensors."""
    configs, n, _ = xya.shape
    x, y, a = xya.unbind(2)
    c, s = torch.cos(a), torch.sin(a)
    sg = lambda v: torch.where(v.abs() > 1e-6, torch.where(v >= 0, 1.0, -1.0), 0.0).to(v.dtype)  # noqa: E731
    r = 0.5 * (c.abs() + s.abs())
    dr = 0.5 * (-sg(c) * s + sg(s) * c)
    L = side[:, None]
    v = [(r - x).clamp_min(0), (x + r - L).clamp_min(0), (r - y).clamp_min(0), (y + r - L).clamp_min(0)]
    energy = sum(t * t for t in v).sum(1)
    grad = torch.stack([2 * (v[1] - v[0]), 2 * (v[3] - v[2]), 2 * (v[0] + v[1] + v[2] + v[3]) * dr], 2)
    step = max(1, 16_000_000 // (n * n))
    for lo in range(0, configs, step):
        hi = min(configs, lo + step)
        d2 = (x[lo:hi, None, :] - x[lo:hi, :, None]) ** 2 + (y[lo:hi, None, :] - y[lo:hi, :, None]) ** 2
        k, i, j = torch.nonzero(torch.triu(d2 < 2.000001, 1), as_tuple=True)
        k = k + lo
        dx, dy = x[k, j] - x[k, i], y[k, j] - y[k, i]
        ci, si, cj, sj = c[k, i], s[k, i], c[k, j], s[k, j]
        cd, sd = ci * cj + si * sj, si * cj - ci * sj
        rad = 0.5 + 0.5 * (cd.abs() + sd.abs())
        deriv = 0.5 * (sg(sd) * cd - sg(cd) * sd)
        ux, uy = torch.stack([ci, -si, cj, -sj]), torch.stack([si, ci, sj, cj])
        proj = dx * ux + dy * uy
        gap, axis = (proj.abs() - rad).max(0)
        hit = gap < 0
        pick = lambda t: t.gather(0, axis[None])[0]  # noqa: E731
        ux, uy, proj = pick(ux), pick(uy), pick(proj)
        sv = torch.where(proj >= 0, 1.0, -1.0).to(proj.dtype)
        turn = sv * (dy * ux - dx * uy)
        own = axis < 2
        z = torch.where(hit, 2 * gap, torch.zeros_like(gap))
        gi = torch.stack([-z * sv * ux, -z * sv * uy, z * (torch.where(own, turn, 0 * turn) - deriv)], 1)
        gj = torch.stack([z * sv * ux, z * sv * uy, z * (torch.where(own, 0 * turn, turn) + deriv)], 1)
        energy.index_add_(0, k, torch.where(hit, gap * gap, 0 * gap))
        grad.view(-1, 3).index_add_(0, k * n + i, gi)
        grad.view(-1, 3).index_add_(0, k * n + j, gj)
    return energy, grad


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind in ("energy", "energy_host"):
        xya, side = sat_microbench(case["configs"], case["n"], seed)
        f = lambda v: torch.from_numpy(v.astype(np.float32).astype(np.float64)).to(dev)  # noqa: E731
        e, g = _exact_energy(f(xya), f(side))
        return dict(energy=e, grad=g)
    if kind == "energy_fp64":
        states, sides = _states(case, seed)
        got = [_exact_energy(torch.from_numpy(q)[None].to(dev), torch.tensor([w], dtype=torch.float64, device=dev))
               for q, w in zip(states, sides)]
        return dict(energy=torch.cat([e for e, _ in got]), grad=torch.cat([g[0] for _, g in got]))
    return None  # the certifier's verdicts and the searches' states have no value of their own in 64 bits
