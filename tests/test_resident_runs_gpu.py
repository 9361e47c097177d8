"""Resident runs (the default kernel choice) against the kernels that read the
fields of every timestep from memory: the same bits."""
import threading

import numpy as np
import pytest

from wipems_gb300 import Batch, CompressedOperator, Engine, Operator, Scene
from wipems_gb300.fdtd import BC_MUR, BC_PEC, BC_PMC, BC_PML

from test_random_gpu import EXT_SEEDS, GRADED_SEEDS, NR_TS, SEEDS, _splits, random_scene, random_scene_ext

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("libs")]


def _scene(n, wall=BC_PEC):
    s = Scene(*[np.arange(k, dtype=float) for k in n], 1e-3)
    s.set_boundary([wall] * 6, [4 if wall == BC_PML else 0] * 6)
    s.set_gauss_excite(20e9, 20e9, 300)
    c = [k // 2 for k in n]
    s.add_excitation(c, [c[0], c[1], c[2] + 1], [0.3, 0.0, 1.0])
    s.add_probe([c[0], c[1], 0], [c[0], c[1], n[2] - 1], 0)
    return s


def _same(a, b):
    sa, sb = a.samples(), b.samples()
    for x, y in zip([*a.fields(), sa.ts, sa.values, sa.energy], [*b.fields(), sb.ts, sb.values, sb.energy]):
        assert x.tobytes() == y.tobytes()


@pytest.mark.parametrize("n,wall", [((21, 21, 21), BC_PEC), ((22, 35, 40), BC_PEC), ((24, 25, 33), BC_PML),
                                    ((23, 20, 26), BC_PMC)])
def test_probes_on_last_lines(n, wall):
    """Probes that read the last line of every axis, which the voltage update
    leaves out at a PEC or UPML wall: current loops around whole
    cross-sections, field probes and voltage lines on it, and what the caller
    wrote there."""
    s = _scene(n, wall)
    top = [k - 1 for k in n]
    for a in range(3):
        lo, hi = [0, 0, 0], list(top)
        lo[a] = hi[a] = n[a] // 3
        s.add_probe(lo, hi, 1, norm_dir=a)
        at = [k // 2 for k in n]
        at[a] = top[a]
        s.add_probe(at, at, 2)
        s.add_probe(at, at, 3)
        line = list(top)
        line[a] = 0
        s.add_probe(line, top, 0)
    s.add_probe(top, top, 2)
    cop = CompressedOperator(Operator(s))
    assert any(p.enabled and max(p.stop[a] == top[a] for a in range(3)) for p in cop.op.probes if p.type == 1)
    es = [Engine(cop, max_timesteps=300, kernel=k) for k in ("auto", "tma")]
    for e in es:
        e.set_frequencies(np.linspace(5e9, 30e9, 3), fd_interval=5)
        e.iterate(20)
        for a in range(3):  # nodes of the probes: on the loops, at the field probe, on the voltage line
            b = (a + 1) % 3
            at = list(top)
            at[a], at[b] = n[a] // 3, n[b] // 2
            e.set_curr(b, *at, 0.125 + a)
            at = [k // 2 for k in n]
            at[a] = top[a]
            e.set_volt(a, *at, -0.5 - a)
            at = list(top)
            at[a] = 3
            e.set_volt(a, *at, 2.0 + a)
        e.iterate(61)
        e.iterate(30)
    _same(*es)
    assert es[0].fd_results()[0].tobytes() == es[1].fd_results()[0].tobytes()
    s = es[1].samples()
    assert np.count_nonzero(np.abs(s.values[s.ts > 25]).max(axis=0) > 0.1) >= 6  # the written values are seen
    for e in es:
        e.close()


@pytest.mark.parametrize("nprobe,interval", [(1, 3), (11, 1), (40, 4)])
def test_samples_without_energies(nprobe, interval):
    """Many samples per run and no energy sums (whose barriers would also
    order the sample rows)."""
    s = _scene((22, 25, 30))
    for k in range(nprobe - 1):
        s.add_probe([k % 21, 12, 0], [k % 21, 12, 29 - k % 5], 0, weight=1.0 + k)
    cop = CompressedOperator(Operator(s))
    es = [Engine(cop, max_timesteps=400, probe_interval=interval, energy_on_probe=False, kernel=k)
          for k in ("auto", "tma")]
    for e in es:
        e.iterate(7)
        e.iterate(200)
    _same(*es)
    assert es[0].samples().values.shape == (207 // interval + 1, nprobe)


@pytest.mark.parametrize("wall,single", [(BC_PEC, 3), (BC_PML, 3), (BC_MUR, 2)])
def test_route_by_length(wall, single):
    """A call of one timestep runs on the half-step kernels (two launches and
    the counter's) unless Mur launches would come beside them; longer calls
    run resident.  Mixed calls give the same bits as the two-pass kernels."""
    cop = CompressedOperator(Operator(_scene((33, 30, 41), wall)))
    es = [Engine(cop, max_timesteps=400, probe_interval=40, kernel=k) for k in ("auto", "tma")]
    launches = {}
    for steps in (1, 1, 2, 1, 30, 1, 1, 64, 1):
        for e in es:
            e.iterate(steps)
        launches.setdefault(steps, set()).add(es[0].last_timing()[1])
    # the first call also takes the sample of numTS 0
    assert launches[1] == {single, single + 1} and launches[2] == {2} and launches[64] <= {2, 3}
    _same(*es)


def test_batched_jobs_hold_no_resident_buffers():
    """Jobs that a batch keeps in its own kernels get no buffers of resident
    runs; a default engine gets them with its first run."""
    cop = CompressedOperator(Operator(_scene((33, 33, 33))))
    for kernel in ("tma", "auto"):
        es = [Engine(cop, max_timesteps=300, kernel=kernel) for _ in range(16)]
        for e in es:
            e.energy()  # nothing to do with stepping
        b0 = Batch(es[:1], bin_mib=64)  # starts the engine: probes and samples
        base = es[0].stats()["device_bytes"]
        b = Batch(es)
        b.iterate(20)
        assert b.stats()["num_bins"] == 1
        assert {e.stats()["device_bytes"] for e in es} == {base}
        es[0].iterate(20)
        assert (es[0].stats()["device_bytes"] > base) == (kernel == "auto")
        for e in (b0, b, *es):
            e.close()


@pytest.mark.parametrize("n,bins", [((130, 128, 120), 0), ((33, 33, 33), 1)])
def test_batch_after_an_asynchronous_iterate(n, bins):
    """A batch takes jobs whose asynchronous steps were not waited for, on
    whichever kernels it steps them."""
    cop = CompressedOperator(Operator(_scene(n)))
    jobs = 2 if bins == 0 else 16
    es, ref = ([Engine(cop, max_timesteps=300, kernel="tma") for _ in range(jobs)] for _ in range(2))
    b = Batch(es)
    assert b.stats()["num_bins"] == bins
    es[0].iterate_async(30)
    b.iterate(20)
    es[0].wait()
    assert [e.num_timesteps for e in es[:2]] == [50, 20]
    for e, steps in zip(ref, (50, 20)):
        e.iterate(steps)
    for e, r in zip(es[:2], ref):
        for x, y in zip(e.fields(), r.fields()):
            assert x.tobytes() == y.tobytes()
    for e in (b, *es, *ref):
        e.close()


def test_interval_graph_of_many_timesteps():
    """A probe interval above 65536 timesteps replays its graph as a shorter
    one does: one chunk's launches, one counter launch."""
    cop = CompressedOperator(Operator(_scene((6, 5, 7))))
    e = Engine(cop, max_timesteps=200000, probe_interval=70000, kernel="tma")
    e.iterate(70000)
    assert e.last_timing()[1] in (2 * 70000 + 1, 2 * 70000 + 2)  # and the sample of numTS 0
    e.iterate(70000)
    assert e.last_timing()[1] == 2 * 70000 + 1 and list(e.samples().ts) == [0, 70000, 140000]


def test_engines_that_share_the_gpu():
    """Asynchronous calls run on the half-step kernels, which overlap; a
    synchronous call runs resident while no other engine has timesteps in
    flight.  Engines on their own streams and threads, resident or not, give
    the bits of one that runs alone."""
    walls = (BC_PEC, BC_PML, BC_MUR, BC_PEC)
    sizes = ((42, 35, 40), (46, 33, 61), (45, 40, 44), (90, 88, 70))
    cops = [CompressedOperator(Operator(_scene(n, w))) for n, w in zip(sizes, walls)]
    ref = [Engine(c, max_timesteps=3000, kernel="tma") for c in cops]
    es = [Engine(c, max_timesteps=3000) for c in cops]
    for e in ref:
        e.iterate(2200)
    for e in es:
        e.iterate_async(100)
    for e in es:
        e.wait()
        assert e.last_timing()[1] > 200
    es[0].iterate_async(50)
    es[1].iterate(50)  # beside the first engine's
    assert es[1].last_timing()[1] > 100
    es[0].wait()
    es[0].iterate(50)
    assert es[0].last_timing()[1] <= 4
    es[1].iterate(50)
    for e in es[2:]:
        e.iterate(100)
        assert e.last_timing()[1] <= 4 * (1 + 100 // (64 * e.interval))
    th = [threading.Thread(target=lambda e=e: [e.iterate(k) for k in (1, 499, 1500)]) for e in es]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for e, r in zip(es, ref):
        assert e.num_timesteps == 2200
        _same(e, r)
    b = es[3]
    b.iterate_async(10)
    b.close()  # an engine that ends with timesteps in flight no longer counts
    es[0].iterate(50)
    assert es[0].last_timing()[1] <= 4
    for launches in (100, 0):  # an asynchronous call counts as alone after one that was
        es[0].iterate_async(50)
        es[0].wait()
        assert (es[0].last_timing()[1] > 100) == bool(launches)
    ref[0].iterate(150)
    _same(es[0], ref[0])


def test_many_engines_with_upml():
    """Engines that join a crowd of four or more run resident where that is the
    faster way for many, with the same bits."""
    cop = CompressedOperator(Operator(_scene((61, 60, 62), BC_PML)))
    es = [Engine(cop, max_timesteps=300) for _ in range(7)]
    ref = Engine(cop, max_timesteps=300, kernel="tma")
    ref.iterate(150)
    for steps in (100, 50):
        for e in es:
            e.iterate_async(steps)
        for e in es:
            e.wait()
    launches = [e.last_timing()[1] for e in es]
    assert min(launches[:3]) > 100 and max(launches[3:]) <= 4, launches
    for e in es:
        _same(e, ref)


@pytest.mark.parametrize("n", [(20, 21, 22), (33, 30, 34), (22, 37, 65)])
def test_one_plane_chunks(n):
    """The current kernel with fewer registers for chunks of one plane (UPML,
    16-bit indices), on sample steps and between."""
    cop = CompressedOperator(Operator(_scene(n, BC_PML)))
    es = [Engine(cop, max_timesteps=300, kernel="tma", x_chunk=1), Engine(cop, max_timesteps=300, kernel="direct")]
    for e in es:
        e.iterate(37)
        e.iterate(120)
    assert es[0].stats()["x_chunk"] == 1
    _same(*es)


@pytest.mark.parametrize("interval,fd,runs", [(0, 0, 3), (3, 0, 11), (7, 0, 5), (3, 1, 11), (0, 1, 9), (11, 5, 3)])
def test_run_splits(interval, fd, runs):
    """One call over the limits of a run: 1024 timesteps, 64 samples and 256
    frequency-domain steps."""
    cop = CompressedOperator(Operator(_scene((22, 25, 30))))
    es = [Engine(cop, max_timesteps=3000, probe_interval=interval, kernel=k) for k in ("auto", "tma")]
    for e in es:
        if fd:
            e.set_frequencies(np.linspace(5e9, 30e9, 3), fd_interval=fd)
        e.iterate(2100)
    per_run = 2 + (interval > 0) + (fd > 0)  # the run, its samples, energies and frequency-domain sums
    initial = (interval > 0) + (fd > 0)      # of numTS 0
    n = es[0].last_timing()[1] - initial
    assert 2 * runs <= n <= per_run * runs, n
    _same(*es)
    if fd:
        assert es[0].fd_results()[0].tobytes() == es[1].fd_results()[0].tobytes()
        assert es[0].fd_results()[1] == 2100 // fd + 1


@pytest.mark.parametrize("n,wall,fits", [((104, 100, 98), BC_PEC, True), ((112, 111, 110), BC_PEC, False),
                                         ((80, 80, 80), BC_PML, True), ((92, 90, 88), BC_PML, False),
                                         ((90, 88, 70), BC_MUR, True), ((104, 101, 99), BC_MUR, False)])
def test_grids_around_the_capacity(n, wall, fits):
    cop = CompressedOperator(Operator(_scene(n, wall)))
    es = [Engine(cop, max_timesteps=300, kernel=k) for k in ("auto", "tma")]
    for e in es:
        e.iterate(40)
    assert (es[0].last_timing()[1] <= 5) == fits
    assert es[1].last_timing()[1] > 80
    _same(*es)


def test_batch_of_resident_jobs():
    cop = CompressedOperator(Operator(_scene((61, 60, 62), BC_PML)))
    es = [Engine(cop, max_timesteps=300, kernel="tma") for _ in range(3)]
    b = Batch(es, x_chunk=64, blocks_per_sm=-1, chains=2)
    assert b.stats()["num_bins"] == 0  # nothing left for the batched kernels
    b.iterate(50)
    assert b.stats()["last_launches"] <= 3 * 3


@pytest.mark.parametrize("seed", SEEDS + GRADED_SEEDS + EXT_SEEDS)
def test_random_scenes_on_the_default_engine(seed):
    """The random sweeps with the engine's own choice of kernels, resident
    where the scene allows, in split runs."""
    ext = seed in EXT_SEEDS
    op = Operator(random_scene_ext(seed) if ext else random_scene(seed, graded=seed in GRADED_SEEDS))
    cop = CompressedOperator(op)
    ref = Engine(cop, kernel="direct")
    ref.iterate(NR_TS)
    eng = Engine(cop)
    rng = np.random.default_rng(4000 + seed)
    for k in _splits(rng, NR_TS):
        eng.iterate(k)
    _same(eng, ref)
    for p in op.probes:
        if p.enabled and p.type in (0, 1):
            assert eng.probe_now(p) == ref.probe_now(p)


@pytest.mark.parametrize("n,wall", [((12, 11, 32), BC_PEC), ((21, 20, 22), BC_PML), ((91, 92, 90), BC_MUR)])
def test_engines_that_always_run_resident(n, wall):
    """Grids so small that the SMs hold several, and large ones with Mur faces."""
    cop = CompressedOperator(Operator(_scene(n, wall)))
    es = [Engine(cop, max_timesteps=300, probe_interval=7) for _ in range(3)]
    ref = Engine(cop, max_timesteps=300, probe_interval=7, kernel="tma")
    ref.iterate(100)
    for e in es:
        e.iterate_async(100)
    for e in es:
        e.wait()
        assert e.last_timing()[1] <= 5
        _same(e, ref)
