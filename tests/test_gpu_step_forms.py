"""GPU parity of the forms a step takes at the edges of their ranges, against
the CPU oracle, bit for bit:
* the walker hash kept at a high load, where its tombstones pile up and it is
  rebuilt inside a call (cleared behind one step, refilled by the next sweep)
  and between calls;
* a spawn list refused for its length between two steps, and a step with more
  attempts than its list holds;
* heavy parents, whose spawn attempts are numbered by the spawn kernel instead
  of written as entries: around the limit, around the granules, alone and
  many side by side;
* lattices with one coupling and with several, the lookup of their children
  in the spawn kernel or behind it, core parents, and walker hashes the
  spawn kernel's table cannot hold."""
from __future__ import annotations

import ctypes
import itertools

import numpy as np
import pytest

from neci_stable_gb300 import capi
from neci_stable_gb300.engine import Engine
from neci_stable_gb300.systems import make_rows
from oracle.oracle import Oracle

from helpers import canonical, hubbard10, hubbard_square, molecule, random_walkers

pytestmark = pytest.mark.gpu


def same_list(spec, eng, orc, tag):
    W, L = spec.W, spec.lenof_sign
    rg, rc = canonical(eng.download()[0], W), canonical(orc.download()[0], W)
    assert rg.shape == rc.shape, tag
    assert np.array_equal(rg[:, :W + L], rc[:, :W + L]), tag
    assert np.array_equal(rg[:, -1] & ~1, rc[:, -1] & ~1), tag


def run_both(spec, eng, orc, calls, tau, seed, shift=0.0):
    """calls[i] steps in the i-th call of the engine, the lists compared
    after every call and the counts after every step."""
    it = 1
    for n in calls:
        p = capi.default_params(tau=tau, diag_sft=[shift, shift], seed=seed, iter=it)
        sg = eng.iterate_n(p, n)
        for k in range(n):
            q = capi.default_params(tau=tau, diag_sft=[shift, shift], seed=seed, iter=it + k)
            sc, rc = orc.iterate(q)
            assert rc == 0 and sg[k].err == 0 and sg[k].reserved == 0, (it + k, rc, sg[k].err)
            for f in ("n_attempts", "n_spawned", "n_unique", "n_new", "n_occupied"):
                assert getattr(sg[k], f) == getattr(sc, f), (f, it + k)
            assert sg[k].n_occupied + sg[k].holes_in_list == sg[k].tot_walkers
        it += n
        same_list(spec, eng, orc, it)


@pytest.mark.parametrize("lenof_sign", [1, 2])
@pytest.mark.parametrize("calls", [(400,), (1,) * 200 + (3,) * 60, (150, 1, 7, 150)])
def test_walker_hash_at_high_load(lenof_sign, calls):
    # the table's length is 2 max_walkers (a power of two): the list in use
    # keeps it 0.4 live, and a turnover of 6% a step piles tombstones up
    spec = hubbard10(lenof_sign=lenof_sign)
    eng = Engine(spec, 1 << 12, 1 << 14)
    orc = Oracle(spec, 1 << 13, 1 << 15, hii=eng.hii)
    eng.start_from_reference(initial_part=900.0 if lenof_sign == 1 else 840.0)
    orc.upload(eng.download()[0])
    run_both(spec, eng, orc, calls, tau=0.02, seed=5, shift=-5.39 if lenof_sign == 1 else -5.4)
    eng.close()


def test_large_walker_hash_rebuilt_inside_a_call():
    # a table that several blocks clear (2^25 buckets): one call of 60 steps,
    # whose determinants take more places of the table than it may hold,
    # against calls of one step, which rebuild it between them.  A determinant
    # missing from the table would be counted as a new one.
    spec = hubbard_square(4, 4, 16)
    half = [sum(1 << 2 * o for o in c) for c in itertools.combinations(range(16), 8)][::12][:1000]
    dets = (np.array(half)[:, None] | (np.array(half)[None, :] << 1)).reshape(-1, 1)
    counts = []
    for last in ((60,), (1,) * 60):
        eng = Engine(spec, 1 << 24, 1 << 24)
        eng.upload(make_rows(dets, np.full(dets.size, 2.0), np.full(dets.size, 1 << 13)))
        stats = []
        for n, shift in [(10, 6.0)] * 6 + [(n, -9.0) for n in last]:
            stats += eng.iterate_n(capi.default_params(tau=0.01, diag_sft=[shift] * 2, seed=6, iter=1 + len(stats)), n)
        assert all(s.err == 0 and s.reserved == 0 for s in stats)
        counts.append([(s.n_occupied, s.n_new, s.n_unique, s.n_spawned, s.n_attempts) for s in stats])
        eng.close()
    assert sum(c[1] for c in counts[0]) > 0.65 * 2 ** 25
    assert counts[0] == counts[1]


def test_hash_after_entry_points_between_steps():
    # the counters and the walker hash an entry point finds between two steps
    spec = molecule(12, 6)
    eng = Engine(spec, 1 << 14, 1 << 16)
    orc = Oracle(spec, 1 << 14, 1 << 16, hii=eng.hii)
    eng.start_from_reference(initial_part=3000.0)
    orc.upload(eng.download()[0])
    run_both(spec, eng, orc, (30,), tau=0.01, seed=9)
    rows = eng.download()[0]
    sp = rows[::3].copy()
    sp[:, spec.W:spec.W + 1] = (-sp[:, spec.W:spec.W + 1].view(np.float64)).view(np.int64)
    for it in (31, 32, 33):
        p = capi.default_params(tau=0.01, seed=9, iter=it)
        sg = eng.annihilate(p, sp)
        sc, rc = orc.annihilate(p, sp)
        assert rc == 0 and sg.err == 0
        same_list(spec, eng, orc, it)
    out_g, _ = eng.compress_spawns(sp)
    assert out_g.shape[0] == np.unique(sp[:, 0]).size
    eng.set_core_space(eng.download()[0][:50, :spec.W])
    gone = np.setdiff1d(rows[:, 0], eng.download()[0][:, 0])
    if gone.size:
        with pytest.raises(capi.NeciGpuError):
            eng.set_core_space(gone[:1, None])


@pytest.mark.parametrize("ann", [capi.ANN_HASH, capi.ANN_SORT])
def test_steps_after_a_refused_spawn_list(ann):
    # a spawn list longer than the capacity is refused before anything is
    # counted: the next steps' free list holds every hole once
    spec = molecule(12, 6)
    eng = Engine(spec, 1 << 13, 1 << 13)
    orc = Oracle(spec, 1 << 13, 1 << 13, hii=eng.hii)
    eng.set_option(capi.OPT_ANNIHILATION, ann)
    eng.start_from_reference(initial_part=600.0)
    orc.upload(eng.download()[0])
    run_both(spec, eng, orc, (40,), tau=0.01, seed=13)
    long_list = np.repeat(eng.download()[0][:1], (1 << 13) + 1, axis=0)
    it = 41
    for _ in range(3):
        with pytest.raises(capi.NeciGpuError) as ei:
            eng.annihilate(capi.default_params(tau=0.01, seed=13, iter=it), long_list)
        assert ei.value.code == capi.ERR_SPAWN_FULL
        with pytest.raises(capi.NeciGpuError) as ei:
            eng.compress_spawns(long_list)
        assert ei.value.code == capi.ERR_SPAWN_FULL
        p = capi.default_params(tau=0.01, seed=13, iter=it)
        sg, (sc, rc) = eng.perform_fcimc_cyc_par(p), orc.iterate(p)
        assert rc == 0 and sg.err == 0 and sg.holes_in_list > 0
        assert abs(sg.tot_parts_old[0] - sc.tot_parts_old[0]) <= 1e-12 * sc.tot_parts_old[0]
        same_list(spec, eng, orc, it)
        it += 1


@pytest.mark.parametrize("name,lenof_sign", [("hub", 1), ("mol", 1), ("mol", 2)])
@pytest.mark.parametrize("big", [0.0, 30.0, 2500.0])
def test_more_attempts_than_the_list_holds(name, lenof_sign, big):
    # entries, heavy parents or both pass the 3072 attempts of the list, in a
    # step behind a list read: the step fails without an attempt, and a list
    # that fits runs again
    spec = hubbard10(lenof_sign=lenof_sign) if name == "hub" else molecule(12, 6, lenof_sign=lenof_sign)
    eng = Engine(spec, 1 << 12, 1 << 10)
    orc = Oracle(spec, 1 << 12, 1 << 12, hii=eng.hii)
    rows = random_walkers(spec, 700, np.random.default_rng(41))
    W, L = spec.W, spec.lenof_sign
    v = rows[:, W:W + L].view(np.float64).copy()
    v[:, :] = 6.0 if big == 0.0 else 1.0
    if big:
        v[: 120 if big < 100.0 else 2, 0] = big
    rows[:, W:W + L] = v.view(np.int64)
    few = rows.copy()
    few[:, W:W + L] = np.ones_like(v).view(np.int64)
    for it in (1, 2):
        eng.upload(rows)
        eng.download()
        st = capi.IterStats()
        p = capi.default_params(tau=0.002, seed=3, iter=it)
        assert eng.lib.neci_gpu_iterate(eng.ctx, ctypes.byref(p), ctypes.byref(st)) == capi.ERR_SPAWN_FULL
        assert st.err == capi.ERR_SPAWN_FULL and st.n_attempts == int(v.sum()) > 3072 and st.n_spawned == 0
        eng.upload(few)
        orc.upload(few)
        eng.download()
        run_both(spec, eng, orc, (2,), tau=0.002, seed=17)


def test_error_of_the_step_behind_an_upload():
    # the upload's reset of the status comes before the step's first kernel
    spec = hubbard10()
    eng = Engine(spec, 1 << 12, 1 << 10)
    rows = random_walkers(spec, 700, np.random.default_rng(44))
    rows[:, spec.W] = np.float64(6.0).view(np.int64)
    p = capi.default_params(tau=0.002, seed=3, iter=1)
    st = capi.IterStats()
    for _ in range(100):
        eng.upload(rows)
        assert eng.lib.neci_gpu_iterate(eng.ctx, ctypes.byref(p), ctypes.byref(st)) == capi.ERR_SPAWN_FULL
        assert st.err == capi.ERR_SPAWN_FULL


@pytest.mark.parametrize("lenof_sign", [1, 2])
@pytest.mark.parametrize("n,rest", [(31, 31.0), (32, 1.0), (32, 40.0), (33, 1.0), (64, 2.0)])
def test_attempts_past_36_bits(lenof_sign, n, rest):
    # n amplitudes of 2^31 (2^31 attempts each): around and past the 2^36
    # attempts that the heavy parents' packed count holds, the step is refused
    # as any other that passes its list
    spec = hubbard10(lenof_sign=lenof_sign)
    eng = Engine(spec, 1 << 12, 1 << 14)
    rows = random_walkers(spec, 300, np.random.default_rng(43))
    W, L = spec.W, spec.lenof_sign
    v = np.ones((len(rows), L))
    v[:20] = rest
    v.ravel()[60:60 + n] = -2.0 ** 31
    rows[:, W:W + L] = v.view(np.int64)
    eng.upload(rows)
    st = capi.IterStats()
    p = capi.default_params(tau=1e-6, seed=3, iter=1)
    assert eng.lib.neci_gpu_iterate(eng.ctx, ctypes.byref(p), ctypes.byref(st)) == capi.ERR_SPAWN_FULL
    assert st.n_attempts == int(np.abs(v).sum()) and st.n_spawned == 0
    v[:] = 1.0
    rows[:, W:W + L] = v.view(np.int64)
    eng.upload(rows)
    assert eng.perform_fcimc_cyc_par(p).n_attempts == v.size


@pytest.mark.parametrize("name,lenof_sign", [("hub", 1), ("hub", 2), ("mol", 1), ("mol", 2)])
@pytest.mark.parametrize("signs", [(32.0, 33.0), (33.0,) * 40, (127.5, 128.0, 129.0, 31.0, 1.0), (40.0, 5000.0, 1.5, 70000.0),
                                   (1.0, 2.0, 31.0)])
def test_heavy_parents(name, lenof_sign, signs):
    spec = hubbard10(lenof_sign=lenof_sign) if name == "hub" else molecule(12, 6, lenof_sign=lenof_sign)
    eng = Engine(spec, 1 << 15, 1 << 18)
    orc = Oracle(spec, 1 << 15, 1 << 18, hii=eng.hii)
    rng = np.random.default_rng(31)
    rows = random_walkers(spec, 300, rng)
    W, L = spec.W, spec.lenof_sign
    v = rows[:, W:W + L].view(np.float64).copy()
    for k, x in enumerate(signs):  # in both runs, of either sign
        v[7 * k, 0] = -x if k % 2 else x
        v[7 * k + 3, L - 1] = x
    rows[:, W:W + L] = v.view(np.int64)
    eng.upload(rows)
    orc.upload(rows)
    run_both(spec, eng, orc, (1, 2), tau=0.002, seed=17)


def lattice(kind, lenof_sign):
    """Lattices the spawn kernel takes in its form for one coupling (ring,
    duplicated neighbours, six neighbours, two words) and in the general one
    (couplings that differ in size or sign)."""
    if kind == "ring":
        return hubbard10(lenof_sign=lenof_sign)
    if kind == "two-wide":  # left and right neighbour are the same site
        return hubbard_square(2, 3, 6, lenof_sign)
    if kind == "6x6":
        return hubbard_square(6, 6, 35, lenof_sign)
    spec = hubbard_square(3, 4, 11, lenof_sign)
    if kind == "triangular":
        nb = np.zeros((12, 6), dtype=np.int32)
        for s in range(12):
            x, y = s % 3, s // 3
            for k, (dx, dy) in enumerate(((-1, 0), (1, 0), (0, -1), (0, 1), (1, 1), (-1, -1))):
                nb[s, k] = (y + dy) % 4 * 3 + (x + dx) % 3 + 1
        nb[5, 2] = 0  # a site with a neighbour less in the middle of its list
    else:
        nb = spec.neighbours
    t = np.zeros((24, 24))
    rng = np.random.default_rng(3)
    for s in range(12):
        for n in nb[s]:
            if n > s + 1:
                v = -1.3 if kind == "triangular" else (rng.choice([-1.0, 1.0]) if kind == "signs" else -rng.uniform(0.3, 2.0))
                for sp in (0, 1):
                    t[2 * s + sp, 2 * n - 2 + sp] = t[2 * n - 2 + sp, 2 * s + sp] = v
    spec.neighbours = nb
    spec.tmat = np.ascontiguousarray(t.T)
    return spec


@pytest.mark.parametrize("kind", ["ring", "two-wide", "6x6", "triangular", "signs", "sizes"])
@pytest.mark.parametrize("lenof_sign,fuse,core,real,prec", [(1, 1, 0, 1, 1), (1, 1, 40, 1, 0), (2, 1, 40, 0, 0), (2, 0, 40, 1, 0),
                                                            (1, 0, 0, 0, 1)])
@pytest.mark.parametrize("big_hash", [False, True])
def test_lattice_spawn_forms(kind, lenof_sign, fuse, core, real, prec, big_hash):
    spec = lattice(kind, lenof_sign)
    if big_hash:  # products with the electron's number leave 32 bits
        spec.random_hash2 = (spec.random_hash2.astype(np.int64) * 40009 % (1 << 31)).astype(np.int32)
    eng = Engine(spec, 1 << 15, 1 << 17)
    orc = Oracle(spec, 1 << 15, 1 << 17, hii=eng.hii)
    eng.set_option(capi.OPT_FUSE_PROBE, fuse)
    rows = random_walkers(spec, 400, np.random.default_rng(8))
    eng.upload(rows)
    orc.upload(rows)
    if core:
        cd = rows[:core, :spec.W]
        eng.set_core_space(cd)
        orc.set_core_space(cd)
    for tau_search in (0, 1):
        eng.set_tau_search(bool(tau_search))
        orc.set_tau_search(bool(tau_search))
        for it in range(1 + 3 * tau_search, 4 + 3 * tau_search):
            p = capi.default_params(tau=0.01, seed=23, iter=it, t_all_real_coeff=real, precision=prec)
            sg = eng.perform_fcimc_cyc_par(p)
            sc, rc = orc.iterate(p)
            assert rc == 0 and sg.err == 0
            for f in ("n_attempts", "n_spawned", "n_unique", "n_new", "n_occupied"):
                assert getattr(sg, f) == getattr(sc, f), (f, it)
            same_list(spec, eng, orc, it)
    a, b = eng.tau_stats(), orc.tau_stats()
    assert a.gamma_sing == b.gamma_sing and a.cnt_sing == b.cnt_sing


@pytest.mark.parametrize("name,lenof_sign,walkers", [("hub", 1, 300), ("mol12", 2, 200), ("mol24", 1, 400), ("mol48", 1, 300),
                                                     ("mol40", 2, 300)])
def test_short_and_long_spawn_lists(name, lenof_sign, walkers):
    # both forms of the annihilation on the same list: the short form until a
    # step writes more records than its lines, the long form after that
    # (determinants of 1, 2 and 3 words, diagonal tables that fit shared
    # memory and that do not)
    spec = hubbard10(lenof_sign=lenof_sign) if name == "hub" else molecule(int(name[3:]), 8, lenof_sign=lenof_sign)
    eng = Engine(spec, 1 << 21, 1 << 22)
    orc = Oracle(spec, 1 << 21, 1 << 22, hii=eng.hii)
    rng = np.random.default_rng(12)
    rows = random_walkers(spec, walkers, rng)
    W, L = spec.W, spec.lenof_sign
    for scale, tau, steps in ((1.0, 0.005, 3), (400.0, 0.02, 2), (1600.0, 0.02, 2)):
        if scale > 400.0 and name not in ("mol24", "mol40"):
            continue
        v = rows[:, W:W + L].view(np.float64) * scale
        r = rows.copy()
        r[:, W:W + L] = np.ascontiguousarray(v).view(np.int64)
        eng.upload(r)
        orc.upload(r)
        for it in range(1, steps + 1):
            p = capi.default_params(tau=tau, seed=29, iter=it)
            sg = eng.perform_fcimc_cyc_par(p)
            sc, rc = orc.iterate(p)
            assert rc == 0 and sg.err == 0
            for f in ("n_attempts", "n_spawned", "n_unique", "n_new", "n_occupied"):
                assert getattr(sg, f) == getattr(sc, f), (f, it, scale)
            same_list(spec, eng, orc, (it, scale))


def form_of_a_step(eng, p):
    """Whether the lookup's kernel compressed the spawns of one step (the
    compression is counted, with no time of its own)."""
    eng.set_profiling(True)
    eng.kernel_times()
    st = eng.perform_fcimc_cyc_par(p)
    kt = eng.kernel_times()
    eng.set_profiling(False)
    assert st.err == 0 and kt["ann_compress"][1] == 1 and kt["ann_probe"][1] == 1 and kt["ann_probe"][0] > 0.0
    return kt["ann_compress"][0] == 0.0


def test_times_of_a_short_spawn_list():
    spec = molecule(24, 8)
    eng = Engine(spec, 1 << 21, 1 << 22)
    rows = random_walkers(spec, 300, np.random.default_rng(12))
    for scale, short in ((1.0, True), (4000.0, False)):
        r = rows.copy()
        r[:, spec.W] = (rows[:, spec.W].view(np.float64) * scale).view(np.int64)
        eng.upload(r)
        p = capi.default_params(tau=0.02, seed=29, iter=1)
        st = eng.perform_fcimc_cyc_par(p)  # chooses the form of the next step
        assert st.n_spawned < 400000 if short else st.n_spawned > 600000, st.n_spawned
        p.iter = 2
        assert form_of_a_step(eng, p) == short


def test_stages_are_counted_once_a_step():
    spec = molecule(12, 6, lenof_sign=2)
    eng = Engine(spec, 1 << 14, 1 << 16)
    eng.start_from_reference(initial_part=300.0)
    eng.set_rdm_sampling(True)
    eng.set_profiling(True)
    eng.kernel_times()
    eng.iterate_n(capi.default_params(tau=0.01, seed=29, iter=1), 7)
    kt = eng.kernel_times()
    for stage in ("sweep", "spawn", "ann_probe", "ann_compress", "ann_insert", "merge_stats", "rdm", "final"):
        assert kt[stage][1] == 7, (stage, kt[stage])
    assert kt["rdm"][0] > 0.0


def test_form_of_the_first_step():
    # a context that has not stepped yet takes the form of its list's length
    spec = molecule(24, 8)
    half = [sum(1 << 2 * o for o in c) for c in itertools.combinations(range(24), 4)][:1200]
    dets = (np.array(half)[:, None] | (np.array(half)[None, :] << 1)).reshape(-1, 1)  # 1.44e6
    p = capi.default_params(tau=0.001, seed=29, iter=1)
    for lengths in ((1000, dets.size), (dets.size, 1000)):
        eng = Engine(spec, 1 << 21, 1 << 22)
        for n in lengths:
            eng.upload(make_rows(dets[:n], np.ones(n), np.zeros(n, dtype=np.int64)))
        assert form_of_a_step(eng, p) == (n == 1000)
        eng.close()


@pytest.mark.parametrize("lenof_sign", [1, 2])
@pytest.mark.parametrize("n,max_spawned", [(1, 4096), (1023, 4096), (1024, 4096), (1025, 700), (5000, 700), (5000, 1500), (5000, 5000)])
def test_download_packs_the_occupied_slots(lenof_sign, n, max_spawned):
    # lists of less and more than a tile and than the spawn buffer, every
    # third slot a hole; slots in order, whatever is asked for beside the rows
    spec = molecule(24, 10, lenof_sign=lenof_sign)
    eng = Engine(spec, 1 << 14, max_spawned)
    rng = np.random.default_rng(n)
    rows = random_walkers(spec, 2 * n + 50, rng)[:n]
    assert rows.shape[0] == n
    W, L = spec.W, spec.lenof_sign
    rows[1::3, W:W + L] = 0
    dh, odh = rng.normal(size=n), rng.normal(size=n)
    eng.upload(rows, dh, odh)
    keep = np.ones(n, dtype=bool)
    keep[1::3] = False
    got, gd, go = eng.download()
    assert np.array_equal(got, rows[keep]) and np.array_equal(gd, dh[keep]) and np.array_equal(go, odh[keep])
    out = np.full((int(keep.sum()), eng.R), -1, dtype=np.int64)
    import ctypes as C
    m = C.c_int64()
    capi.check(eng.lib.neci_gpu_download_walkers(eng.ctx, capi.ptr(out), None, None, out.shape[0], C.byref(m)))
    assert m.value == out.shape[0] and np.array_equal(out, rows[keep])
    if out.shape[0] > 1:
        with pytest.raises(capi.NeciGpuError):
            eng.download(max_rows=out.shape[0] - 1)
    eng.start_from_reference(20.0)  # the spawn buffers serve steps as before
    st = eng.iterate_n(capi.default_params(tau=0.001, seed=1, iter=1), 3)
    assert all(x.err == 0 and x.n_attempts > 0 for x in st)
    eng.close()


@pytest.mark.parametrize("lenof_sign", [1, 2])
def test_download_of_amplitudes_at_the_edges(lenof_sign):
    # listed: |C| >= 1e-12 in some run, infinities among them; not: smaller
    # ones, zeros of either sign, NaN
    spec = molecule(12, 6, lenof_sign=lenof_sign)
    eng = Engine(spec, 1 << 12, 1 << 12)
    rows = random_walkers(spec, 200, np.random.default_rng(3))
    W, L = spec.W, spec.lenof_sign
    edge = np.array([1.0, 1e-12, np.nextafter(1e-12, 0.0), -1e-12, 0.0, -0.0, np.nan, -np.nan, np.inf, -np.inf, 5e-324])
    v = np.zeros((len(rows), L))
    v[:, 0] = edge[np.arange(len(rows)) % edge.size]
    v[:, L - 1] = edge[np.arange(len(rows)) % edge.size if L == 1 else np.arange(len(rows)) // edge.size % edge.size]
    rows[:, W:W + L] = v.view(np.int64)
    eng.upload(rows)
    with np.errstate(invalid="ignore"):
        listed = (np.abs(v) >= 1e-12).any(axis=1)
    assert np.array_equal(eng.download()[0][:, :W + L], rows[listed][:, :W + L])
    eng.set_core_space(rows[listed][:30, :W])
    assert np.array_equal(eng.download()[0][:, :W + L], rows[listed][:, :W + L])


@pytest.mark.parametrize("n_ctx", [7, 8, 33, 68])
def test_batch_with_smaller_grids(n_ctx):
    # the grids of a batch's contexts shrink from 8 contexts on, down to the
    # fewest blocks (a short capacity) and to several rounds a block
    from neci_stable_gb300.engine import iterate_batch
    specs = [hubbard10(), molecule(12, 6), hubbard10(lenof_sign=2)]
    walkers = [random_walkers(sp, 2000, np.random.default_rng(60 + k), scale=4.0) for k, sp in enumerate(specs)]
    params = [capi.default_params(tau=0.004, seed=70 + i, iter=1) for i in range(n_ctx)]

    def fresh(i):
        e = Engine(specs[i % 3], 1 << (13 if i % 2 else 17), 1 << (15 if i % 2 else 18))
        e.upload(walkers[i % 3])
        return e

    batch = [fresh(i) for i in range(n_ctx)]
    iterate_batch(batch, params, 6)
    for i in range(0, n_ctx, 1 if n_ctx < 10 else 5):
        alone = fresh(i)
        alone.iterate_n(params[i], 6)
        W = specs[i % 3].W
        assert np.array_equal(canonical(batch[i].download()[0], W), canonical(alone.download()[0], W)), i


@pytest.mark.parametrize("n_ctx,sizes", [(16, (17, 12, 12)), (33, (18, 12, 15)), (64, (17, 13, 13))])
def test_batch_of_uneven_contexts(n_ctx, sizes):
    # the first context's capacity is 4 to 64 times the others': its grids
    # shrink by its part of the batch, theirs by their number
    from neci_stable_gb300.engine import iterate_batch
    specs = [molecule(14, 8), hubbard10(lenof_sign=2), molecule(12, 6)]
    walkers = [random_walkers(specs[0], 20000, np.random.default_rng(80), scale=2.0)]
    walkers += [random_walkers(sp, 900, np.random.default_rng(81 + k), scale=4.0) for k, sp in enumerate(specs[1:])]
    params = [capi.default_params(tau=0.004, seed=170 + i, iter=1) for i in range(n_ctx)]

    def fresh(i):
        k = 0 if i == 0 else 1 + i % 2
        e = Engine(specs[k], 1 << sizes[k], 1 << sizes[k] + 1)
        e.upload(walkers[k])
        return e, specs[k].W

    batch = [fresh(i)[0] for i in range(n_ctx)]
    iterate_batch(batch, params, 5)
    for i in (0, 1, 2, n_ctx - 1):
        alone, W = fresh(i)
        alone.iterate_n(params[i], 5)
        assert np.array_equal(canonical(batch[i].download()[0], W), canonical(alone.download()[0], W)), i


@pytest.mark.parametrize("n", [1, 31, 257, 1500])
def test_sums_of_the_sweeps(n):
    # the sweeps' sums in fixed point: amplitudes around its limits (2048 for
    # the population, 128 for the deaths, which the shift makes large, small
    # and negative), against sums without rounding.  A term is off by at most
    # 2^-53 (population) or 2^-57 (deaths), the FP64 sum of the blocks' sums
    # by a few units in its last place.
    import math
    spec = hubbard10()
    rng = np.random.default_rng(90 + n)
    rows = random_walkers(spec, n, rng)
    W = spec.W
    edge = np.array([2047.9999999999998, 2048.0, 2048.0000000000005, 1.0, 1.0000000000000002, 0.7, 3.3e5, 1e-3, 2.0 ** -40])
    amp = np.where(np.arange(len(rows)) % 3 == 0, rng.choice(edge, len(rows)), rng.lognormal(0.0, 2.0, len(rows)))
    amp *= rng.choice([-1.0, 1.0], len(rows))
    rows[:, W] = amp.view(np.int64)
    eng = Engine(spec, 1 << 17, 1 << 25)  # up to 2e7 attempts
    for shift in (-2.0, 0.0, 9.0):
        eng.upload(rows)
        held, dh, _ = eng.download()
        c = np.ascontiguousarray(held[:, W]).view(np.float64)
        fac = 0.01 * (dh - shift)
        died = [min(f * abs(x), abs(x)) for f, x in zip(fac, c)]
        p = capi.default_params(tau=0.01, diag_sft=[shift, shift], seed=4, iter=1)
        st = eng.perform_fcimc_cyc_par(p)
        assert st.err == 0
        for got, terms, unit in ((st.tot_parts_old[0], np.abs(c).tolist(), 2.0 ** -53), (st.ndied[0], died, 2.0 ** -57)):
            size = math.fsum(abs(t) for t in terms)
            assert abs(got - math.fsum(terms)) <= len(terms) * unit + 16 * 2.0 ** -53 * size, (shift, got)
        after = np.ascontiguousarray(eng.download()[0][:, W]).view(np.float64)
        total = math.fsum(np.abs(after))
        assert abs(st.tot_parts[0] - total) <= len(after) * 2.0 ** -53 + 16 * 2.0 ** -53 * total


@pytest.mark.parametrize("n", [30, 3000])
@pytest.mark.parametrize("tau,low,high", [(1e-7, -6.0, 0.0), (1e-4, -9.0, -6.0), (1e-4, -1.0, 4.0), (1e-9, 3.0, 9.0)])
def test_sums_of_the_sweeps_relative(n, tau, low, high):
    # the sweeps' sums of amplitudes of any size keep the precision of FP64
    # sums: a sum of terms t is off by at most 40 roundings of its partial
    # sums (two terms a thread, sixteen additions over a block, an addition
    # for each of a dozen blocks), 40 x 2^-53 sum |t|
    import math
    spec = hubbard10()
    rng = np.random.default_rng(n)
    rows = random_walkers(spec, n, rng)
    W = spec.W
    amp = 10.0 ** rng.uniform(low, high, len(rows)) * rng.choice([-1.0, 1.0], len(rows))
    if high > 8.0:
        amp[3:] = 1.0 + rng.uniform(0.0, 1.0, len(rows) - 3)  # few large ones: their attempts fit
        amp[:3] *= 1e-3
    rows[:, W] = amp.view(np.int64)
    eng = Engine(spec, 1 << 14, 1 << 23)

    def near(got, terms):
        terms = [float(t) for t in terms]
        assert abs(got - math.fsum(terms)) <= 40 * 2.0 ** -53 * math.fsum(abs(t) for t in terms), got

    def signs():
        held, dh, _ = eng.download()
        o = np.argsort(held[:, 0])
        return held[o, 0], np.ascontiguousarray(held[o, W]).view(np.float64), dh[o]

    for core in (False, True):
        for shift in (-3.0, 6.0):
            eng.upload(rows)
            if core:
                eng.set_core_space(rows[:, :W])
            dets, c, dh = signs()
            fac = tau * (dh - shift)
            died = np.minimum(fac * np.abs(c), np.abs(c))
            st = eng.perform_fcimc_cyc_par(capi.default_params(tau=tau, diag_sft=[shift, shift], seed=4, iter=1))
            near(st.tot_parts_old[0], np.abs(c))
            near(st.ndied[0], died)
            dets1, c1, _ = signs()
            near(st.tot_parts[0], np.abs(c1))
            if not core and st.n_spawned == 0:
                left = np.abs(c - died * np.sign(c))
                rounded = left < 1.0
                stays = np.isin(dets, dets1)
                near(st.nremoved[0], left[rounded & ~stays])
                near(st.nborn[0], 1.0 - left[rounded & stays])


def same_rdm(eng, orc, tag):
    # atomic FP64 sums on both sides of the comparison: their order is free
    a, b = eng.rdm2(), orc.rdm2()
    np.testing.assert_allclose(a, b, rtol=1e-9, atol=1e-12 * max(np.abs(b).max(), 1.0), err_msg=str(tag))


@pytest.mark.parametrize("batch", [False, True])
def test_rdm_of_a_call_that_fails(batch):
    # a call of many steps whose eleventh has more attempts than the list
    # holds: the steps up to it leave both parts of their 2-RDM, as one-step
    # calls do, and so does the call after the next upload
    from neci_stable_gb300.engine import iterate_batch
    spec = molecule(12, 6, lenof_sign=2)

    def fresh(max_spawned):
        e = Engine(spec, 1 << 14, max_spawned)
        e.start_from_reference(initial_part=3000.0)
        e.set_rdm_sampling(True)
        e.rdm2(reset=True)
        return e

    def params(it):
        return capi.default_params(tau=0.01, diag_sft=[2.0, 2.0], seed=8, iter=it)

    free = fresh(1 << 16)
    start = free.download()[0]
    attempts = [free.perform_fcimc_cyc_par(params(it)).n_attempts for it in range(1, 21)]
    fail = next(k for k in range(10, 20) if attempts[k] > max(attempts[:k]) + 2)
    room = (max(attempts[:fail]) - 1024) // 2 + 1
    one, many = fresh(room), fresh(room)
    with pytest.raises(capi.NeciGpuError):
        for it in range(1, 21):
            one.perform_fcimc_cyc_par(params(it))
    assert it == fail + 1
    with pytest.raises(capi.NeciGpuError) as ei:
        if batch:
            iterate_batch([many, free], [params(1), params(21)], 20)
        else:
            many.iterate_n(params(1), 20)
    assert ei.value.code == capi.ERR_SPAWN_FULL
    same_rdm(many, one, "after the failed call")
    for e in (one, many):
        e.upload(start)
    many.iterate_n(params(1), 5)
    for it in range(1, 6):
        one.perform_fcimc_cyc_par(params(it))
    same_rdm(many, one, "after the next call")


@pytest.mark.parametrize("name,pop,core,batch,calls", [("hub", 300.0, 0, False, (2, 7, 30)), ("hub", 300.0, 30, True, (7, 1, 12)),
                                                       ("mol12", 400.0, 0, True, (2, 7, 30)), ("mol12", 400.0, 40, False, (2, 7, 30)),
                                                       ("mol33", 400.0, 0, False, (3, 9)), ("mol24", 0.0, 0, False, (2, 3))])
def test_rdm_of_calls_of_several_steps(name, pop, core, batch, calls):
    # the diagonal summed per slot over a call: slots freed and filled again,
    # emptied by the annihilation, core slots, both forms of the annihilation
    # (mol24 passes the lines of the short one), one and two words
    from neci_stable_gb300.engine import iterate_batch
    big = name == "mol24"
    shift = [-5.4] * 2 if name == "hub" else [0.0] * 2  # the ring's population would outgrow its list
    spec = hubbard10(lenof_sign=2) if name == "hub" else molecule(int(name[3:]), 8 if big else 6, lenof_sign=2)
    cap = (1 << 21, 1 << 22) if big else (1 << 15, 1 << 17)
    eng, other, orc = Engine(spec, *cap), Engine(spec, *cap), None
    orc = Oracle(spec, *cap, hii=eng.hii)
    if big:
        rows = random_walkers(spec, 300, np.random.default_rng(5))
        rows[:, spec.W:spec.W + 2] = (rows[:, spec.W:spec.W + 2].view(np.float64) * 1000.0).view(np.int64)
        eng.upload(rows)
    else:
        eng.start_from_reference(initial_part=pop)
        eng.iterate_n(capi.default_params(tau=0.02, diag_sft=shift, seed=2, iter=1), 20)
    rows = eng.download()[0]
    for e in (eng, other, orc):
        e.upload(rows)
        if core:
            o = np.argsort(-np.abs(rows[:, spec.W:spec.W + 2].view(np.float64)).sum(axis=1), kind="stable")
            e.set_core_space(rows[o[:core], :spec.W])
        e.set_rdm_sampling(True)
        e.rdm2(reset=True)
    it, removed, placed, spawned = 1, 0.0, 0, 0
    for n in calls:
        p = capi.default_params(tau=0.02, diag_sft=shift, seed=6, iter=it)
        if batch:
            stats = iterate_batch([other, eng], [p, p], n)[0][1]
        else:
            stats = eng.iterate_n(p, n)
        for k in range(n):
            sc, rc = orc.iterate(capi.default_params(tau=0.02, diag_sft=shift, seed=6, iter=it + k))
            assert rc == 0 and stats[k].err == 0 and stats[k].n_occupied == sc.n_occupied
            removed += stats[k].nremoved[0] + stats[k].nremoved[1]
            placed += stats[k].n_new
            spawned = max(spawned, stats[k].n_spawned)
        it += n
        same_list(spec, eng, orc, it)
        same_rdm(eng, orc, it)
        if batch:
            same_rdm(other, orc, it)
    assert removed > 0.0 and placed > 0 and (spawned > 600000) == big
