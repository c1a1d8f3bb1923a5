"""The work this framework is used for, as cases that can be timed and compared.

A case is one system (a Hubbard lattice or a synthetic molecule), a walker
population and a way of calling the engine; a pass is what the host program
around the engine does between two of its own decisions: one call of
PerformFCIMCycPar, a cycle of StepsSft iterations with its shift update, a
batch of instances, a stretch of 2-RDM sampling, a restart leg between two
POPSFILEs, or a deterministic projection.  The population a case starts from is grown by the host loop
(`fcimc.FciMCPar`) on the device, from the seed alone.

A pass returns every number of every iteration's statistics record
(`neci_gpu_iter_stats`), which is all the iteration hands its caller while the
walker list stays resident, and the walker list itself where the program reads
it back.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from neci_stable_gb300 import capi, systems
from neci_stable_gb300.engine import Engine, iterate_batch
from neci_stable_gb300.fcimc import CalcParams, FciMCPar

FLOATS = ("nborn", "ndied", "nannihil", "naborted", "nremoved", "tot_parts", "tot_parts_old", "noat_hf", "hf_cyc",
          "enum_cyc", "norm_psi_sq")
COUNTS = ("n_occupied", "n_attempts", "n_spawned", "n_unique", "n_new", "n_core")
STATS = np.dtype([(k, "f8", (2,)) for k in FLOATS] +
                 [(k, "i8") for k in ("tot_walkers", "n_occupied", "holes_in_list", "n_attempts", "n_spawned",
                                      "n_unique", "n_new", "n_core")] + [("err", "i4"), ("reserved", "i4")])

# What a case is when it does not say otherwise.
DEFAULTS = dict(call="cycle", steps=10, precision="fp64", replicas=1, rdm=False, core=0, gen="pchb", real=True,
                ann="hash", ms2=0, tau=0.0, equil=200, settle=60, scale=1.0, slots=3.0, spawns=4.0, dets=0.2, instances=0)


def listed():
    return [
        # The smallest call: the host's own loop calls PerformFCIMCycPar once
        # per iteration on the 10-site ring (1e4 walkers, 3e3 determinants);
        # a step is a dozen short launches, so latency counts.
        dict(name="ring10_one_step", system="chain", lx=10, nel=10, walkers=1e4, tau=0.01, call="iterate", steps=1,
             equil=400, slots=20.0, spawns=100.0, dets=0.34),
        # The whole space of the same ring as the deterministic space: 10
        # projections per pass (63504 rows, 6e5 elements), then the vector is
        # read back.  The deterministic part of every semistochastic run.
        dict(name="ring10_full_core", system="chain", lx=10, nel=10, walkers=1e5, tau=0.01, call="project", steps=10,
             dets=0.63504, slots=2.0, spawns=2.0),
        # A small molecule with the uniform generator and integer walkers,
        # the defaults of an input that names neither PCHB nor real
        # coefficients (the size of NECI's own Ne test).
        dict(name="n14_uniform_integer", system="molecule", n=14, nel=8, walkers=5e4, gen="uniform", real=False,
             equil=600, slots=10.0, spawns=10.0, dets=0.21),
        # A restart leg of an ordinary run: the POPSFILE's rows are uploaded,
        # a cycle runs, the rows are read back for the next POPSFILE.
        dict(name="n24_restart_leg", system="molecule", n=24, nel=10, walkers=1e6, call="restart", dets=0.29),
        # The benchmark molecule at its stated size, in FP64 ...
        dict(name="n24_fp64", system="molecule", n=24, nel=10, walkers=1e7, dets=0.143),
        # ... and with FP32 spawn amplitudes.
        dict(name="n24_mixed", system="molecule", n=24, nel=10, walkers=1e7, precision="mixed", dets=0.143),
        # The sort form of the annihilation, which NECI itself uses and the
        # autotuner tries.
        dict(name="n24_sort", system="molecule", n=24, nel=10, walkers=2e6, ann="sort", dets=0.24),
        # One replica pair sampling the 2-RDM in every step, the sums read (and
        # begun again) after five cycles; n = 32 has a second, empty
        # determinant word.
        dict(name="n32_replicas_rdm", system="molecule", n=32, nel=12, walkers=3e5, replicas=2, rdm=True, call="rdm",
             steps=50, slots=8.0,
             spawns=8.0, dets=0.83),
        # The batch configuration: 64 instances of uneven size (n 12..40, 1e4
        # to 1e6 walkers) side by side, replica pairs sampling the 2-RDM, FP32
        # amplitudes.
        dict(name="batch64_rdm_mixed", system="molecule", call="batch", instances=64, walkers=1e5, replicas=2, rdm=True,
             precision="mixed", tau=0.005, equil=100, slots=8.0, spawns=8.0, dets=0.3),
        # An open-shell molecule with an odd electron count and two words.
        dict(name="n39_odd_open_shell", system="molecule", n=39, nel=15, ms2=1, walkers=3e6, dets=0.43),
        # The 6x6 lattice with a semistochastic core: many determinants, many
        # spawns per slot.
        dict(name="hub6x6_core", system="square", lx=6, ly=6, nel=36, walkers=4e7, tau=0.003, core=10_000,
             equil=260, scale=20.0, slots=2.0, spawns=2.0, dets=0.66),
        # The largest molecule, three words a row, semistochastic core, mixed
        # precision, at a fifth of its stated population.
        dict(name="n64_core_mixed", system="molecule", n=64, nel=20, walkers=1e8, tau=0.002, core=50_000,
             precision="mixed", equil=600, scale=20.0, slots=0.8, spawns=1.0, dets=0.48),
    ]


def draw(rng):
    """One more case of the same ranges: a lattice or a molecule of any size
    between the smallest and the largest, walkers spread over their
    logarithm, and the options the listed cases use."""
    kind = rng.choice(["chain", "square", "molecule", "molecule", "molecule"])
    walkers = float(round(10 ** rng.uniform(4.0, 7.0 if kind == "molecule" else 6.5)))
    c = dict(system=kind, walkers=walkers, replicas=rng.choice([1, 1, 2]),
             precision=rng.choice(["fp64", "mixed"]), ann=rng.choice(["hash", "hash", "hash", "sort"]),
             call=rng.choice(["iterate", "cycle", "cycle", "restart" if walkers < 3e6 else "cycle"]))
    if kind == "chain":
        c["lx"] = rng.randint(10, 36)
    elif kind == "square":
        c["lx"], c["ly"] = rng.choice([(3, 4), (4, 4), (5, 4), (5, 5), (6, 5), (6, 6)])
    else:
        c["n"] = rng.randint(12, 40)
        c["nel"] = rng.randint(6, min(20, c["n"]))
        c["ms2"] = c["nel"] % 2
        c["gen"] = rng.choice(["pchb", "pchb", "pchb", "uniform"])
        c["real"] = rng.choice([True, True, True, False])
    if kind != "molecule":
        sites = c["lx"] * c.get("ly", 1)
        c["nel"] = sites - rng.choice([0, 0, 1, 2, 3])
        c.update(tau=round(0.1 / sites, 5), equil=240, slots=12.0, spawns=12.0, dets=0.55)
    else:
        c.update(slots=8.0 if walkers < 1e6 else 4.0, spawns=8.0 if walkers < 1e6 else 4.0, dets=0.4)
        if c["gen"] == "uniform":
            c["equil"] = 600
        if c["replicas"] == 2:
            c["rdm"] = rng.choice([True, False])
        if c.get("rdm"):
            c.update(call="rdm", steps=50)
    if c["call"] == "iterate":
        c["steps"] = 1
    if walkers >= 1e5 and not c.get("rdm") and rng.random() < 0.3:
        c["core"] = rng.choice([500, 2000, 10_000])
    return c


def full(case):
    return {**DEFAULTS, **case}


@functools.lru_cache(maxsize=4)
def integrals(n, seed):
    """The synthetic FCIDUMP of n orbitals: a file on disk in a user's run."""
    return systems.synthetic_fcidump(n, seed)


def spec_of(c, seed):
    if c["system"] != "molecule":
        dims = (c["lx"],) if c["system"] == "chain" else (c["lx"], c["ly"])
        return systems.hubbard_system(c["system"], dims, c["nel"], u=4.0, seed=seed % 1000 + 7,
                                      lenof_sign=c["replicas"])
    h, eri, ecore = integrals(c["n"], 20240601 + c["n"])
    return systems.molecular_system(h, eri, ecore, c["nel"], ms2=c["ms2"], seed=seed % 1000 + 7,
                                    lenof_sign=c["replicas"],
                                    excitgen=capi.EXGEN_PCHB if c["gen"] == "pchb" else capi.EXGEN_UNIFORM)


def engine_of(c, spec):
    eng = Engine(spec, max_walkers=int(max(c["slots"] * c["walkers"], 2e5)),
                 max_spawned=int(max(c["spawns"] * c["walkers"], 4e5)))
    if c["ann"] == "sort":
        eng.set_option(capi.OPT_ANNIHILATION, capi.ANN_SORT)
    return eng


def grow(c, eng, seed):
    """The population of the case, grown by the host loop of FciMCPar: a
    lattice from a few walkers with the shift held until the target is
    reached, a molecule from the target number on its reference with the
    conventional tau search (unless tau is given), the shift varying.  The
    list is then scaled to the target, as in a restart from a rescaled
    POPSFILE, and settles (large ones are grown at 1 / scale of the target)."""
    lattice = c["system"] != "molecule"
    target = c["walkers"] / c["scale"]
    calc = CalcParams(tau=c["tau"] or 0.002, target_walkers=target, sft_damp=0.5, seed=seed,
                      precision=capi.PREC_FP64, all_real_coeff=c["real"], tau_search=not c["tau"],
                      tau_search_max_iter=c["equil"] // 2)
    drv = FciMCPar(eng, calc)
    if lattice:
        eng.start_from_reference(initial_part=max(20.0, 0.002 * target))
    else:
        eng.start_from_reference(initial_part=target)
        drv.single_part_phase = [False] * eng.L
    res = drv.run(c["equil"])
    if drv.single_part_phase[0]:
        raise RuntimeError(f"the population did not reach its target in {c['equil']} iterations")
    factor = c["walkers"] / res.tot_parts[-1]
    if not c["real"]:
        factor = max(1, round(factor))
    rows, dh, odh = eng.download(max_rows=int(eng.csys.max_walkers))
    W, L = eng.W, eng.L
    rows[:, W:W + L] = (rows[:, W:W + L].view(np.float64) * factor).view(np.int64)
    eng.upload(rows, dh, odh)
    drv.run(c["settle"])
    if c["core"]:
        rows, _, _ = eng.download(max_rows=int(eng.csys.max_walkers))
        eng.set_core_space(most_populated(rows, c["core"], W, L), capi.PREC_FP64)
        drv.run(10)
    calc.precision = capi.PREC_MIXED if c["precision"] == "mixed" else capi.PREC_FP64
    if c["rdm"]:
        eng.set_rdm_sampling(True)
    return drv


def most_populated(rows, n, words, runs):
    """pops-core: the n determinants of largest weight, those of equal weight
    in the order of their determinants."""
    r = by_determinant(rows, words)
    weight = r[:, words:words + runs].contiguous().view(torch.float64).abs().sum(1)
    return r[torch.argsort(weight, descending=True, stable=True)[:n], :words].cpu().numpy()


def ring_sector(nsites, nel):
    """Every determinant of the ring's Sz = 0 sector as one word each, spin
    orbital p (1-based; odd beta, even alpha) at bit p - 1, in a fixed order."""
    nhalf = nel // 2
    masks = np.array([m for m in range(1 << nsites) if bin(m).count("1") == nhalf], dtype=np.int64)
    spread = np.zeros(masks.size, dtype=np.int64)
    for s in range(nsites):
        spread |= ((masks >> s) & 1) << (2 * s)
    return (spread[:, None] | (spread[None, :] << 1)).ravel()


def ring_start(c, seed):
    """The deterministic projection's start: each determinant's walkers fall
    off with its number of doubly occupied sites, with a random sign."""
    dets = ring_sector(c["lx"], c["nel"])
    pairs = dets & (dets >> 1) & 0x5555555555555555
    docc = np.array([bin(x).count("1") for x in pairs.tolist()])
    rng = np.random.default_rng(seed)
    v = rng.normal(0.0, 1.0, dets.size) * np.exp(-0.8 * docc)
    return dets, docc, v * (c["walkers"] / np.abs(v).sum())


RING_SHIFT = -5.83434  # the ring's ground-state energy, where its shift settles


def prepare(case, seed):
    c = full(case)
    if c["call"] == "batch":
        return prepare_batch(c, seed)
    spec = spec_of(c, seed)
    eng = engine_of(c, spec)
    if c["call"] == "project":
        dets, _, v = ring_start(c, seed)
        eng.upload(systems.make_rows(dets[:, None], v, np.full(dets.size, 1 << 13)))
        eng.set_core_space(dets[:, None], capi.PREC_FP64)
        params = capi.default_params(tau=c["tau"], diag_sft=[RING_SHIFT], seed=seed, iter=1)
        return dict(case=c, eng=eng, params=params, n=dets.size)
    drv = grow(c, eng, seed)
    state = dict(case=c, eng=eng, drv=drv, params=drv.params(), old=None)
    if c["call"] == "restart":
        rows, dh, odh = eng.download(max_rows=int(c["slots"] * c["walkers"] + 2e5))
        state.update(rows=rows.copy(), diag=dh.copy(), offdiag=odh.copy())
        if c["core"]:
            state["core"] = most_populated(rows, c["core"], eng.W, eng.L)
    return state


def prepare_batch(c, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(7000)  # the molecules: n 12..40, 6..20 electrons, uneven populations
    engines, params = [], []
    for i in range(c["instances"]):
        n = int(sizes.integers(12, 41))
        nel = min(int(2 * sizes.integers(3, 11)), n - n % 2)
        walkers = c["walkers"] * float(10 ** sizes.uniform(-1.0, 1.0))
        one = {**c, "n": n, "nel": nel, "walkers": walkers}
        eng = engine_of(one, spec_of(one, seed + i))
        eng.start_from_reference(initial_part=walkers)
        eng.set_rdm_sampling(c["rdm"])
        engines.append(eng)
        params.append(capi.default_params(tau=c["tau"], seed=int(rng.integers(1 << 40)), iter=1))
    state = dict(case=c, engines=engines, params=params, old=[None] * len(engines))
    for _ in range(c["equil"] // 10):
        batch_cycle(state, 10, 0.5)
    for p in params:
        p.precision = capi.PREC_MIXED if c["precision"] == "mixed" else capi.PREC_FP64
    return state


def batch_cycle(state, n, damp):
    stats, _ = iterate_batch(state["engines"], state["params"], n)
    for i, (p, st) in enumerate(zip(state["params"], stats)):
        p.iter += n
        state["old"][i] = vary_shift(p, st, state["old"][i], damp)
    return stats


def vary_shift(p, stats, old, damp):
    """update_shift of a cycle, on the parameters the next call gets."""
    parts = list(stats[-1].tot_parts)
    old = old or list(stats[0].tot_parts_old)
    for k in range(2):
        if parts[k] > 0.0 and old[k] > 0.0:
            p.diag_sft[k] -= damp * math.log(parts[k] / old[k]) / (p.tau * len(stats))
    return parts


def records(stats, runs):
    """The statistics records as arrays, one row an iteration."""
    a = np.frombuffer(b"".join(bytes(s) for s in stats), dtype=STATS)
    out = {k: np.ascontiguousarray(a[k][:, :runs]) for k in FLOATS}
    out.update({k: np.ascontiguousarray(a[k]) for k in COUNTS})
    return out


def by_determinant(rows, words):
    """Downloaded rows in the order of their determinants (a list has none of
    its own), sorted on the device as a program that compares lists does."""
    r = torch.from_numpy(rows).cuda()
    for w in reversed(range(words)):
        r = r[torch.argsort(r[:, w], stable=True)]
    return r


def split_rows(r, words, runs, room):
    """Determinants and signs of sorted rows in a program's own buffers of
    `room` rows, unused ones zero."""
    dets = torch.zeros((room, words), dtype=torch.int64, device=r.device)
    signs = torch.zeros((room, runs), dtype=torch.float64, device=r.device)
    dets[:r.shape[0]] = r[:, :words]
    signs[:r.shape[0]] = r[:, words:words + runs].contiguous().view(torch.float64)
    return dets, signs


def run(state):
    c, call = state["case"], state["case"]["call"]
    if call == "batch":
        stats = batch_cycle(state, c["steps"], 0.05)
        return records([s for per in stats for s in per], 2)
    eng, p = state["eng"], state["params"]
    if call == "iterate":
        st = eng.perform_fcimc_cyc_par(p)
        p.iter += 1
        if p.iter % 10 == 0:
            state["old"] = vary_shift(p, [st] * 10, state["old"], 0.1)
        return records([st], eng.L)
    if call == "cycle":
        stats = eng.iterate_n(p, c["steps"])
        p.iter += c["steps"]
        state["old"] = vary_shift(p, stats, state["old"], 0.1)
        return records(stats, eng.L)
    if call == "rdm":
        stats = []
        for _ in range(c["steps"] // 10):
            stats += eng.iterate_n(p, 10)
            p.iter += 10
            state["old"] = vary_shift(p, stats[-10:], state["old"], 0.1)
        return dict(rdm2=eng.rdm2(reset=True), stats=records(stats, eng.L))
    if call == "project":
        stats = eng.iterate_n(p, c["steps"])
        rows, _, _ = eng.download(max_rows=state["n"])
        W, L = eng.W, eng.L
        return dict(dets=rows[:, :W], signs=np.ascontiguousarray(rows[:, W:W + L]).view(np.float64),
                    stats=records(stats, L))
    # restart: the list is put back, a cycle runs from it, the list is read
    eng.upload(state["rows"], state["diag"], state["offdiag"])
    if c["core"]:
        eng.set_core_space(state["core"], capi.PREC_FP64)
    stats = eng.iterate_n(p, c["steps"])
    room = int(1.25 * c["walkers"] * c["replicas"]) + 1000
    rows, _, _ = eng.download(max_rows=room)
    dets, signs = split_rows(by_determinant(rows, eng.W), eng.W, eng.L, room)
    return dict(dets=dets, signs=signs, stats=records(stats, eng.L))


def exact(case, seed):
    """The deterministic projection in plain numpy: C <- C - tau (H - S) C on
    the ring's sector.  The other cases are one realisation of a stochastic
    process whose draws are the framework's own counter-based streams: they
    have no value of their own outside it."""
    c = full(case)
    if c["call"] != "project":
        return None
    dets, docc, v = ring_start(c, seed)
    order = np.argsort(dets, kind="stable")
    srt = dets[order]
    cols, rows, vals = [], [], []
    nsites = c["lx"]
    for s in range(nsites):
        t = (s + 1) % nsites
        for spin in (0, 1):
            a, b = 2 * s + spin, 2 * t + spin
            src = np.nonzero(((dets >> a) & 1 == 1) & ((dets >> b) & 1 == 0))[0]
            child = dets[src] ^ (1 << a) ^ (1 << b)
            lo, hi = min(a, b), max(a, b)
            between = (dets[src] >> (lo + 1)) & ((1 << (hi - lo - 1)) - 1)
            odd = np.array([bin(x).count("1") & 1 for x in between.tolist()])
            dst = order[np.searchsorted(srt, child)]
            el = np.where(odd == 1, 1.0, -1.0)  # t = 1, b = -t
            for i, j in ((src, dst), (dst, src)):
                rows.append(i)
                cols.append(j)
                vals.append(el)
    rows, cols, vals = (np.concatenate(x) for x in (rows, cols, vals))
    parts = [np.abs(v).sum()]
    norm = []
    for _ in range(c["steps"]):
        y = np.bincount(rows, weights=vals * v[cols], minlength=v.size)
        v = v - c["tau"] * ((4.0 * docc - RING_SHIFT) * v + y)
        parts.append(np.abs(v).sum())
        norm.append((v * v).sum())
    none = {k: None for k in FLOATS + COUNTS}
    return dict(dets=None, signs=v[:, None],
                stats={**none, "tot_parts": np.array(parts[1:])[:, None],
                       "tot_parts_old": np.array(parts[:-1])[:, None], "norm_psi_sq": np.array(norm)[:, None]})


def work(case):
    """Per iteration: the walker list read and written once (det words, signs,
    flag word, two diagonal elements), per spawn attempt two multiplies of its
    amplitude and, for a molecule, half an integral sum; per determinant the
    death step; a 2-RDM is read once.  A projection reads the core Hamiltonian (8 B value, 4 B
    column) and the vector and writes the vector.  A list that the program
    uploads and reads back moves once each way more."""
    c = full(case)
    L = c["replicas"]
    if c["call"] == "batch":
        sizes = np.random.default_rng(7000)
        total = {"bytes": 0.0, "flops": 0.0}
        for _ in range(c["instances"]):
            n = int(sizes.integers(12, 41))
            nel = min(int(2 * sizes.integers(3, 11)), n - n % 2)
            walkers = c["walkers"] * float(10 ** sizes.uniform(-1.0, 1.0))
            one = work({**c, "call": "cycle", "n": n, "nel": nel, "walkers": walkers})
            total = {k: total[k] + one[k] for k in total}
        return total
    nbasis = 2 * (c["n"] if c["system"] == "molecule" else c["lx"] * c.get("ly", 1))
    words = nbasis // 64 + 1
    row = 8 * (words + L + 1)
    dets = c["dets"] * c["walkers"]
    if c["call"] == "project":
        nnz = 11.1 * dets
        step = 12 * nnz + 16 * dets
        return {"bytes": float(c["steps"] * step + 16 * dets), "flops": float(c["steps"] * (2 * nnz + 4 * dets))}
    attempts = c["walkers"] * L
    per_attempt = 2 + (c["nel"] / 2 if c["system"] == "molecule" else 4)
    data = c["steps"] * dets * (2 * row + 16) + (2 * dets * (row + 16) if c["call"] == "restart" else 0)
    if c["call"] == "rdm":
        data += 8 * (nbasis * (nbasis - 1) // 2) ** 2
    return {"bytes": float(data), "flops": float(c["steps"] * (attempts * per_attempt + 5 * dets * L))}
