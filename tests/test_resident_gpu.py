"""Grids that fit in shared memory run resident (the default kernel choice):
fields, samples, energies and frequency-domain sums must equal the direct
kernels bit for bit, at extents around the 32-node segments and the box
cuts, with and without UPML, trimmed and untrimmed last lines, graded
meshes, Mur faces, lumped RLC, Drude and Lorentz bricks, and through split runs, field writes and restores."""
import numpy as np
import pytest

from wipems_gb300 import Batch, CompressedOperator, Engine, Operator, Scene
from wipems_gb300.fdtd import BC_MUR, BC_PEC, BC_PMC, BC_PML

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("libs")]


def _op(n, wall=BC_PEC, graded=False, media=()):
    rng = np.random.default_rng(sum(n))
    lines = [np.cumsum(rng.uniform(0.8, 1.2, k)) if graded else np.arange(k, dtype=float) for k in n]
    s = Scene(*lines, 1e-3)
    walls = wall if isinstance(wall, list) else [wall] * 6
    s.set_boundary(walls, [4 if w == BC_PML else 0 for w in walls])
    s.set_gauss_excite(20e9, 20e9, 300)
    c = [k // 2 for k in n]
    at = lambda *i: [lines[a][min(i[a], n[a] - 1)] for a in range(3)]
    s.add_excitation(at(*c), at(c[0], c[1], c[2] + 1), [0.3, 0.0, 1.0])
    if min(n) > 8:
        s.add_material(at(c[0] - 2, c[1] - 3, 5), at(c[0] + 2, c[1] + 1, c[2] + 2), eps_r=3.0, kappa=0.2, priority=10)
    if "rlc" in media:
        for k in range(2):
            s.add_lumped_rlc(at(c[0] - 3, c[1] + 2 + k, c[2]), at(c[0] - 3, c[1] + 2 + k, c[2] + 1), 2, R=50.0, L=2e-9,
                             Cap=0.5e-12, series=False, caps=False, priority=1000)
    for k, m in enumerate(("drude", "lorentz")):
        if m in media:
            s.add_lorentz(at(c[0] + 1, 3, 4 + 6 * k), at(c[0] + 4, c[1] - 4, 9 + 6 * k), eps_r=2.0, plasma_f=[9e9],
                          relax_t=[1e-9], pole_f=[6e9 if k else 0.0], mue_plasma_f=[5e9], mue_relax_t=[1e-9],
                          priority=20 + k)
    s.add_probe(at(c[0], c[1], 0), at(c[0], c[1], n[2] - 1), 0)
    return Operator(s)


def _same(a, b):
    sa, sb = a.samples(), b.samples()
    for x, y in zip([*a.fields(), sa.ts, sa.values, sa.energy], [*b.fields(), sb.ts, sb.values, sb.energy]):
        assert x.tobytes() == y.tobytes()


_MIX = [BC_MUR, BC_MUR, BC_PEC, BC_MUR, BC_MUR, BC_PMC]


@pytest.mark.parametrize("n,wall,graded,media", [
    ((3, 3, 3), BC_PEC, False, ()), ((2, 9, 40), BC_PEC, False, ()), ((6, 35, 2), BC_PMC, False, ()),
    ((33, 9, 65), BC_PMC, False, ()), ((34, 33, 97), BC_PEC, True, ()), ((20, 21, 22), BC_PML, False, ()),
    ((41, 33, 64), BC_PML, False, ()), ((30, 29, 35), BC_PML, True, ()), ((104, 100, 98), BC_PEC, False, ()),
    ((33, 34, 35), BC_MUR, False, ()), ((22, 31, 65), _MIX, False, ("rlc",)), ((40, 25, 33), BC_MUR, True, ("rlc",)),
    ((21, 22, 40), BC_PML, False, ("rlc",)), ((30, 26, 37), BC_MUR, False, ("drude",)),
    ((30, 27, 64), _MIX, False, ("drude", "lorentz")), ((29, 28, 36), BC_PML, False, ("drude", "lorentz")),
    ((28, 30, 33), BC_PEC, False, ("lorentz", "rlc")), ((30, 31, 38), BC_PML, True, ("drude", "lorentz")),
    ((33, 26, 35), BC_MUR, True, ("drude",)), ((27, 31, 36), BC_PEC, True, ("lorentz",))])
def test_resident_equals_direct(n, wall, graded, media):
    cop = CompressedOperator(_op(n, wall, graded, media))
    a, b = Engine(cop, max_timesteps=300), Engine(cop, max_timesteps=300, kernel="direct")
    if n[0] < 50:
        for e in (a, b):
            e.set_frequencies(np.linspace(5e9, 30e9, 5), fd_interval=7)
    for steps in (1, 2, 40, 83, 100):
        a.iterate(steps)
        b.iterate(steps)
    _same(a, b)
    if n[0] < 50:
        assert a.fd_results()[0].tobytes() == b.fd_results()[0].tobytes() and a.fd_results()[1] == b.fd_results()[1]


def test_resident_writes_and_restore():
    """Fields written by the caller (on the lines no timestep changes too), a
    checkpoint restored to an earlier timestep, and a reset."""
    cop = CompressedOperator(_op((22, 35, 40)))
    a, b = Engine(cop, max_timesteps=300), Engine(cop, max_timesteps=300, kernel="direct")
    for e in (a, b):
        e.iterate(31)
        e.set_volt(2, 10, 12, 20, 0.25)
        e.set_curr(0, 5, 33, 38, -0.5)
        e.set_curr(1, 20, 34, 39, 0.125)
    blob = a.checkpoint()
    for e in (a, b):
        e.iterate(50)
    _same(a, b)
    a.restore(blob)
    a.iterate(50)
    _same(a, b)
    for e in (a, b):
        e.reset()
        e.iterate(45)
    _same(a, b)


@pytest.mark.parametrize("sizes", [[(20, 21, 22)] * 3, [(104, 100, 98), (130, 128, 120), (30, 31, 33)]])
def test_batch_jobs_outside_the_batched_kernels(sizes):
    """Batches whose jobs run resident or on their own kernels: the same
    samples (none before the first timestep of a batch after a reset) and
    fields as L2 bins, which keep every job in the batched kernels."""
    cops = [CompressedOperator(_op(n, BC_PML if k % 2 else BC_PEC)) for k, n in enumerate(sizes)]
    out = []
    for kw in (dict(x_chunk=64, blocks_per_sm=-1, chains=2), dict(bin_mib=64)):
        es = [Engine(c, max_timesteps=300, kernel="tma") for c in cops]
        b = Batch(es, graph_steps=8, **kw)
        b.iterate(21)
        for e in es:
            e.reset()
        b.iterate(50)
        out.append(es)
    for x, y in zip(*out):
        assert x.num_timesteps == y.num_timesteps == 50
        _same(x, y)
