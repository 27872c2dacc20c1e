"""The calls that programs make of this library, as cases that can be timed and compared.

listed() names them, draw() gives more of the same ranges, prepare() makes what a program holds before the call,
run() is one call (or one chunk of a resident run), work() the bytes and operations it cannot do without, exact() the
energies in 64 bits where a call's outputs are pose energies.

The kinds:
  dock      the drop-in call sequence SetParaT / CopyH2D / Dock on one Complex in page-locked memory, Records kept
  ensemble  a resident ensemble of one complex advanced by a chunk of steps and an exchange sweep, states read back
  screen    the same for many ligands of uneven sizes against one pocket
  serve     requests of different ligand sizes sent to a request loop with resident pockets, all results awaited
  poses     energies of many poses with a resident complex
  rescore   energies of a few poses of a Complex, nothing resident
  noalloc   energies of poses whose buffers and Complex are already on the GPU

Monte Carlo chunks are kept short, so that an output holds few Metropolis decisions: one decision that falls the other
way by a rounding changes everything a replica does after it.
"""

import ctypes as C
import math

import numpy as np
import torch

from geauxdock_b200 import dock, layout, params, synth, workmodel
from geauxdock_b200._lib import check, load

FP32, KAHAN, FP64 = 0, 1, 2


def _dock(name, L, P, K, M, nlig, nprt, ntmp, steps, exchange=0):
    return {"name": name, "kind": "dock", "atoms": L, "points": P, "kde": K, "mcs": M, "nlig": nlig, "nprt": nprt,
            "ntmp": ntmp, "steps": steps, "exchange": exchange}


def _ensemble(name, L, P, K, M, nlig, nprt, ntmp, steps, exchange=0, precision=KAHAN, warps=1):
    return dict(_dock(name, L, P, K, M, nlig, nprt, ntmp, steps, exchange), kind="ensemble", precision=precision,
                warps=warps)


def _poses(name, kind, L, P, K, M, nlig, nprt, n, precision):
    return {"name": name, "kind": kind, "atoms": L, "points": P, "kde": K, "mcs": M, "nlig": nlig, "nprt": nprt,
            "poses": n, "precision": precision}


def listed():
    return [
        # one complex, one conformation, one temperature: an interactive docking of one ligand, the smallest Dock call
        _dock("dock_1_replica", 24, 600, 200, 8, 1, 1, 1, 200),
        # the reference's published run: a ligand's 51 conformers against one protein, 100 steps
        _dock("dock_51_replicas", 34, 344, 454, 11, 51, 1, 1, 100),
        # the replica ensemble of 20 ligand x 11 protein conformations x 16 temperatures through Dock
        _dock("dock_3520_replicas", 40, 1500, 400, 16, 20, 11, 16, 10, 10),
        # the same ensemble resident on the GPU, one chunk and its exchange sweep: the long production run's inner call
        _ensemble("ensemble_3520", 40, 1500, 400, 16, 20, 11, 16, 10, 10),
        # a resident single replica in latency mode, 8 warps on it
        _ensemble("ensemble_1_latency", 24, 600, 200, 8, 1, 1, 1, 400, warps=8),
        # an ensemble in FP64 arithmetic, as one checks a long run with
        _ensemble("ensemble_880_fp64", 40, 1500, 400, 16, 20, 11, 4, 3, precision=FP64),
        # uneven ligands of 12-64 atoms against one pocket, 400 replicas each
        {"name": "screen_32_ligands", "kind": "screen", "ligands": 32, "lo": 12, "hi": 64, "points": 2000, "kde": 600,
         "mcs": 16, "nlig": 10, "nprt": 5, "ntmp": 8, "steps": 4, "exchange": 4},
        # a few requests at a time to the request loop, ligands of 8-80 atoms, two resident pockets
        {"name": "serve_4_requests", "kind": "serve", "requests": 4, "lo": 8, "hi": 80, "points": 800, "points2": 2200,
         "kde": 600, "mcs": 16, "nlig": 10, "nprt": 5, "ntmp": 8, "steps": 20, "exchange": 20},
        # rescoring many poses of a large ligand in a large pocket, FP32 and FP64
        _poses("poses_16k_fp32", "poses", 64, 3000, 1000, 16, 1, 1, 16384, FP32),
        _poses("poses_2k_fp64", "poses", 64, 3000, 1000, 16, 1, 1, 2048, FP64),
        # rescoring a handful of poses of one Complex, everything packed for the call
        _poses("rescore_64", "rescore", 40, 1500, 400, 16, 20, 11, 64, FP32),
        # energies of device-resident poses inside another program's GPU work
        _poses("noalloc_4k", "noalloc", 40, 1500, 400, 16, 20, 11, 4096, FP32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dock", "ensemble", "screen", "serve", "poses", "rescore", "noalloc"])
    L, P = _log(rng, 8, 64), _log(rng, 150, 2048)
    K, M = _log(rng, 20, 1000), _log(rng, 1, 40)
    if kind in ("dock", "ensemble"):
        nlig, nprt, ntmp = _log(rng, 1, 30), _log(rng, 1, 11), _log(rng, 1, 16)
        n = nlig * nprt * ntmp
        steps = max(2, min(200, 20000 // n))
        exchange = rng.choice([0, max(2, steps // 2)])
        if kind == "dock":
            c = _dock("", L, P, K, M, nlig, nprt, ntmp, steps, exchange)
        else:
            precision = rng.choice([FP32, KAHAN, KAHAN, FP64])
            c = _ensemble("", L, P, K, M, nlig, nprt, ntmp, max(2, steps // 8) if precision == FP64 else steps,
                          exchange if precision != FP64 else 0, precision, rng.choice([1, 1, 2, 4, 8]))
    elif kind == "screen":
        lo = rng.randrange(8, 30)
        c = {"kind": "screen", "ligands": _log(rng, 2, 32), "lo": lo, "hi": rng.randrange(lo + 1, 81),
             "points": _log(rng, 300, 2400), "kde": K, "mcs": M, "nlig": rng.randrange(1, 11), "nprt": rng.randrange(1, 6),
             "ntmp": rng.randrange(1, 9), "steps": rng.randrange(2, 5), "exchange": 2}
    elif kind == "serve":
        lo = rng.randrange(8, 30)
        steps = rng.randrange(5, 21)
        c = {"kind": "serve", "requests": rng.randrange(1, 5), "lo": lo, "hi": rng.randrange(lo + 1, 81),
             "points": _log(rng, 300, 1000), "points2": _log(rng, 1000, 2200), "kde": K, "mcs": M,
             "nlig": rng.randrange(1, 11), "nprt": rng.randrange(1, 6), "ntmp": rng.randrange(1, 9), "steps": steps,
             "exchange": rng.choice([0, steps // 2])}
    else:
        precision = rng.choice([FP32, FP32, KAHAN, FP64])
        nlig, nprt = _log(rng, 1, 20), _log(rng, 1, 11)
        top = {"poses": 16384, "rescore": 512, "noalloc": 4096}[kind] // (8 if precision == FP64 else 1)
        c = _poses("", kind, L, P, K, M, nlig, nprt, _log(rng, 1, top), precision)
    c.pop("name", None)
    return c


# --------------------------------------------------------------- inputs
_ENEPARA = []


def _enepara():
    if not _ENEPARA:
        _ENEPARA.append(params.optimize_enepara(params.default_enepara0()))
    return _ENEPARA[0]


def _complex_parts(case, seed):
    """Pocket and job of the one-complex kinds."""
    rng = np.random.default_rng(seed)
    pk = synth.make_pocket(rng, case["points"], case["nprt"])
    ntmp = case.get("ntmp", 1)
    temps = synth.ladder(ntmp, 0.3, 3.0) if ntmp > 1 else [0.3]
    job = synth.make_job(rng, pk, case["atoms"], case["nlig"], case["kde"], case["mcs"], temps, seed=seed)
    return pk, job


def _pose_list(case, seed):
    rng = np.random.default_rng(seed + 1)
    n = case["poses"]
    conf = np.stack([rng.integers(0, case["nlig"], n), rng.integers(0, case["nprt"], n)], axis=1).astype(np.int32)
    return conf, synth.config4_poses(seed + 2, n, 6.0)


def _many(case, seed):
    """Pockets and jobs of the screen and serve kinds."""
    rng = np.random.default_rng(seed)
    sizes = [case["points"]] + ([case["points2"]] if "points2" in case else [])
    pockets = [synth.make_pocket(rng, p, case["nprt"]) for p in sizes]
    temps = synth.ladder(case["ntmp"], 0.3, 3.0) if case["ntmp"] > 1 else [0.3]
    jobs = []
    for j in range(case.get("ligands", case.get("requests"))):
        if case["kind"] == "serve":
            L = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        else:
            L = int(rng.integers(case["lo"], case["hi"] + 1))
        p = int(rng.integers(len(pockets)))
        jobs.append(synth.make_job(rng, pockets[p], L, case["nlig"], case["kde"], case["mcs"], temps,
                                   seed=seed + 1000 * (j + 1), pocket_index=p))
    return pockets, jobs


class _State:
    """What a program holds; the library's handles are closed with it."""

    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)

    def __del__(self):
        for k in ("session", "ensemble", "server"):
            h = self.__dict__.pop(k, None)
            if h is not None:
                h.close()


def _pinned(dtype, n=1):
    t = torch.zeros(dtype.itemsize * n, dtype=torch.uint8, pin_memory=True)
    return t, np.frombuffer(t.numpy(), dtype=dtype, count=n)


def _with_options(options, make):
    """make() with process-wide options set for the objects it creates, then set back."""
    lib = load()
    before = {k: lib.gd_get_option(k) for k in options}
    try:
        for k, v in options.items():
            check(lib.gd_set_option(k, v))
        return make()
    finally:
        for k, v in before.items():
            check(lib.gd_set_option(k, v))


def prepare(case, seed):
    kind, ep = case["kind"], _enepara()
    if kind in ("screen", "serve"):
        pockets, jobs = _many(case, seed)
        if kind == "serve":
            return _State(case, server=dock.Server(pockets, ep), jobs=jobs)
        ens = dock.Ensemble.from_jobs(pockets, jobs, ep)
        ens.init()
        ens.sync()
        return _State(case, ensemble=ens)
    pk, job = _complex_parts(case, seed)
    if kind == "poses":
        conf, mm = _pose_list(case, seed)
        return _State(case, ensemble=dock.Ensemble.from_jobs([pk], [job], ep), conf=conf, mm=mm)
    cx = synth.to_complex(job, pk, ep, case.get("steps", 200), case.get("steps", 200), case.get("exchange", 0))
    if kind == "dock":
        keep, work = _pinned(layout.COMPLEX)
        work[0] = cx[0]
        keep_rec, rec = _pinned(layout.RECORD, int(cx[0]["size"]["n_rep"]))
        n = int(cx[0]["size"]["n_rep"])
        return _State(case, session=dock.DockSession(1, seed=seed), cx=work, record=rec, keep=(keep, keep_rec), n=n,
                      start=cx[0]["replica"][:n].copy(), seed=seed)
    if kind == "ensemble":
        ens = _with_options({b"precision": case["precision"], b"replica_warps": case["warps"]},
                            lambda: dock.Ensemble.from_complexes([cx], [seed]))
        ens.init()
        ens.sync()
        return _State(case, ensemble=ens)
    conf, mm = _pose_list(case, seed)
    if kind == "rescore":
        return _State(case, cx=cx, conf=conf, mm=mm)
    dev = torch.from_numpy(cx.view(np.uint8).reshape(-1).copy()).cuda()
    n = case["poses"]
    return _State(case, cx=dev, conf=torch.from_numpy(conf).cuda(), mm=torch.from_numpy(mm).cuda(),
                  out=torch.zeros((n, 10), device="cuda"), raw=torch.zeros((n, 9), device="cuda"))


def _states(r):
    return {f: r[f] for f in ("movematrix", "energy", "step", "is_accept")}


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "dock":
        # the next complex of a queue, with its own seed; the caller's Record array is used again
        s.cx[0]["replica"][:s.n] = s.start
        s.session.seed(s.seed)
        rec = s.session.dock(s.cx, s.record)
        entries = rec["replica"][:, :case["steps"] + 1]
        return {"replicas": _states(s.cx[0]["replica"][:s.n]), "next_entry": rec["next_entry"],
                "records": _states(entries)}
    if kind in ("ensemble", "screen"):
        s.ensemble.run(case["steps"], case["exchange"])
        s.ensemble.sync()
        got = [s.ensemble.replicas(j) for j in range(s.ensemble.njob)]
        st = [s.ensemble.stats(j) for j in range(s.ensemble.njob)]
        if len(got) == 1:
            return {"replicas": _states(got[0]), "stats": st[0]}
        return {"replicas": _states(np.concatenate(got)), "stats": np.concatenate(st)}
    if kind == "serve":
        tickets = [s.server.submit(j, case["steps"], case["exchange"]) for j in s.jobs]
        done = {}
        while len(done) < len(tickets):
            for r in s.server.poll():
                done[r["ticket"]] = r
        rs = [done[t] for t in tickets]
        return {"status": np.array([r["status"] for r in rs]),
                "replicas": _states(np.concatenate([r["replicas"] for r in rs])),
                "stats": np.concatenate([r["stats"] for r in rs])}
    if kind == "poses":
        e, raw, e64 = s.ensemble.eval_poses(0, s.conf, s.mm, case["precision"], want64=case["precision"] == FP64,
                                            want_raw=True)
        return {"energy": e, "raw": raw, "energy64": e64}
    if kind == "rescore":
        e, raw, e64 = dock.eval_poses(s.cx, s.conf, s.mm, case["precision"], want64=case["precision"] == FP64)
        return {"energy": e, "raw": raw, "energy64": e64}
    stream = torch.cuda.current_stream().cuda_stream
    check(load().gd_eval_poses_noalloc(C.c_void_p(s.cx.data_ptr()), case["poses"], C.c_void_p(s.conf.data_ptr()),
                                       C.c_void_p(s.mm.data_ptr()), case["precision"], C.c_void_p(s.out.data_ptr()),
                                       C.c_void_p(s.raw.data_ptr()), C.c_void_p(stream)))
    return {"energy": s.out, "raw": s.raw}


# ----------------------------------------------------------------- work
def _job_bytes(job):
    return (16 * job.lig_xyz.shape[0] * job.natom + 16 * len(job.kde_type) + 16 * len(job.mcs_tcc) * job.natom
            + 4 * job.psp.size)


def work(case):
    """The reference's formulas once per pose (geauxdock_b200/workmodel.py); each input array read once, each state,
    Record entry or energy written once."""
    ep = _enepara()
    if case["kind"] in ("screen", "serve"):
        pockets, jobs = _many(case, 1)
    else:
        pk, job = _complex_parts(case, 1)
        pockets, jobs = [pk], [job]
    per = [workmodel.job_flops_per_pose(j, pockets[j.pocket], ep) for j in jobs]
    data = sum(28 * p.npoint * p.nconf for p in pockets) + sum(_job_bytes(j) for j in jobs)
    if "poses" in case:
        n = case["poses"]
        out = n * (32 + 76 + (80 if case["precision"] == FP64 and case["kind"] != "noalloc" else 0))
        whole = layout.COMPLEX.itemsize if case["kind"] == "rescore" else data
        return {"bytes": whole + out, "flops": n * per[0]}
    n = case["nlig"] * case["nprt"] * case["ntmp"]
    evals = case["steps"] + (0 if case["kind"] in ("ensemble", "screen") else 1)  # the initial energies
    states = len(jobs) * n * (2 * layout.REPLICA.itemsize + 64)
    if case["kind"] == "dock":
        data = layout.COMPLEX.itemsize + n * layout.REPLICA.itemsize
    return {"bytes": data + states, "flops": sum(per) * n * evals}


# ---------------------------------------------------------------- exact
def exact(case, seed):
    """The pose energies in 64 bits (torch on the GPU), from the formulas; None for the Monte Carlo kinds, whose outputs
    depend on every decision before them."""
    if "poses" not in case:
        return None
    pk, job = _complex_parts(case, seed)
    conf, mm = _pose_list(case, seed)
    ep = _enepara()
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def t(a, dtype=torch.float64):
        return torch.as_tensor(np.ascontiguousarray(a), device=dev).to(dtype)

    par = {k: t(np.nan_to_num(np.asarray(ep[k]), nan=0.0, posinf=0.0, neginf=0.0))
           for k in ("p1a", "p2a", "pmf0", "pmf1", "hdb0", "hdb1", "hpl0", "hpl1", "hpl2", "a_para", "b_para", "w")}
    lj0, lj1, el0, el1, a1, b1, kde2, kde3 = (float(ep[k]) for k in ("lj0", "lj1", "el0", "el1", "a1", "b1", "kde2",
                                                                       "kde3"))
    lt, pt = t(job.lig_type, torch.int64), t(pk.type, torch.int64)
    L, M = job.natom, len(job.mcs_tcc)
    tab = {k: par[k][lt][:, pt] for k in ("p1a", "p2a", "pmf0", "pmf1", "hdb0", "hdb1")}
    bonded = tab["hdb0"] > float(np.float32(0.1))
    cls2 = t(pk.cls, torch.int64) == 2
    psp = t(job.psp)[lt][:, t(np.where(pk.cls == 2, pk.seq3r, 0), torch.int64)] * cls2
    hpp = t(pk.hpp) * (t(pk.cdc, torch.int64) == 1)
    q, pe = t(job.lig_charge), t(pk.ele)
    kt = t(job.kde_type, torch.int64)
    match = (lt[:, None] == kt[None, :]).double()
    weight = match / match.sum(1, keepdim=True).clamp(min=1)
    mcs = t(job.mcs_xyz)
    valid = mcs[:, :, 0] != float(layout.MCS_INVALID_COORD)
    tcc = t(job.mcs_tcc)
    pxyz, pcen, lxyz, lcen, kxyz = t(pk.xyz), t(pk.center), t(job.lig_xyz), t(job.lig_center), t(job.kde_xyz)
    cf, mv = t(conf, torch.int64), t(mm)
    raws = []
    step = max(1, 8_000_000 // (L * max(pk.npoint, len(job.kde_type), M)))
    for b in range(0, len(conf), step):
        m, il, ip = mv[b:b + step], cf[b:b + step, 0], cf[b:b + step, 1]
        (s1, s2, s3), (c1, c2, c3) = torch.sin(m[:, 3:]).T, torch.cos(m[:, 3:]).T
        R = torch.stack([c1 * c2, c1 * s2 * s3 - c3 * s1, s1 * s3 + c1 * c3 * s2,
                         c2 * s1, c1 * c3 + s1 * s2 * s3, c3 * s1 * s2 - c1 * s3, -s2, c2 * s3, c2 * c3], 1).view(-1, 3, 3)
        x = torch.einsum("nij,naj->nai", R, lxyz[il]) + (m[:, :3] + lcen[il])[:, None, :]

        def dist2(y):
            return sum((x[:, :, None, k] - y[..., k]) ** 2 for k in range(3))

        d2 = dist2(pxyz[ip][:, None])
        d = d2.sqrt()
        p1, p2 = tab["p1a"] / (d2 ** 4 * d), tab["p2a"] / d2 ** 3
        vdw = ((p1 - p2) / (p1 * lj0 * (1 + lj1 * d2) + 1)).sum((1, 2))
        s = el1 * d
        ele = (q[:, None] * pe * torch.where(s < 1, el0 + a1 * s ** 2 + b1 * s ** 3, 1 / s)).sum((1, 2))
        pmf = (tab["pmf1"] / (1 + torch.exp((-0.5 * d + 6) * (d - tab["pmf0"])))).sum((1, 2))
        pspe = (psp * (d <= tab["pmf0"])).sum((1, 2))
        h = (d - tab["hdb0"]) * tab["hdb1"]
        hdb = torch.where(bonded, tab["hdb1"] * torch.exp(-0.5 * h * h), torch.zeros_like(d)).sum((1, 2))
        z = d2 / 81
        contact = (hpp * torch.where(z <= 1, 1 - 3.5 * z + 4.5 * z ** 2 - 2.5 * z ** 3 + 0.5 * z ** 4,
                                     torch.zeros_like(z))).sum(2)
        hh = (contact - par["hpl0"][lt]) / par["hpl1"][lt]
        hpc = (0.5 * hh * hh - par["hpl2"][lt]).sum(1)
        kde = (weight * torch.exp(kde2 * dist2(kxyz))).sum((1, 2)) / kde3
        sq = sum((x[:, None, :, k] - mcs[None, :, :, k]) ** 2 for k in range(3)) * valid
        lhm = torch.log((tcc * (sq.sum(2) / valid.sum(1)).sqrt()).sum(1) / M)
        dst = (lcen[il] + m[:, :3] - pcen[ip]).square().sum(1).sqrt()
        raws.append(torch.stack([vdw, ele, pmf, pspe, hdb * (-1 / math.sqrt(2 * math.pi)), hpc, kde, lhm, dst], 1))
    raw = torch.cat(raws)
    per = torch.cat([raw[:, :7] / L, raw[:, 7:]], 1)
    e = par["a_para"][:9] * per + par["b_para"][:9]
    e = torch.cat([e, (e * par["w"][:9]).sum(1, keepdim=True)], 1)
    got = {"energy": e.cpu().numpy(), "raw": raw.cpu().numpy()}
    if case["kind"] != "noalloc":
        got["energy64"] = e.cpu().numpy() if case["precision"] == FP64 else None
    return got
