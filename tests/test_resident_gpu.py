"""Grids that fit in shared memory run resident (the default kernel choice):
fields, samples, energies and frequency-domain sums must equal the direct
kernels bit for bit, at extents around the 32-node segments and the box
cuts, with and without UPML, trimmed and untrimmed last lines, graded
meshes, and through split runs, field writes and restores."""
import numpy as np
import pytest

from wipems_gb300 import CompressedOperator, Engine, Operator, Scene
from wipems_gb300.fdtd import BC_PEC, BC_PMC, BC_PML

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("libs")]


def _op(n, wall=BC_PEC, graded=False):
    rng = np.random.default_rng(sum(n))
    lines = [np.cumsum(rng.uniform(0.8, 1.2, k)) if graded else np.arange(k, dtype=float) for k in n]
    s = Scene(*lines, 1e-3)
    s.set_boundary([wall] * 6, [4] * 6 if wall == BC_PML else [0] * 6)
    s.set_gauss_excite(20e9, 20e9, 300)
    c = [k // 2 for k in n]
    at = lambda *i: [lines[a][min(i[a], n[a] - 1)] for a in range(3)]
    s.add_excitation(at(*c), at(c[0], c[1], c[2] + 1), [0.3, 0.0, 1.0])
    if min(n) > 8:
        s.add_material(at(c[0] - 2, c[1] - 3, 5), at(c[0] + 2, c[1] + 1, c[2] + 2), eps_r=3.0, kappa=0.2, priority=10)
    s.add_probe(at(c[0], c[1], 0), at(c[0], c[1], n[2] - 1), 0)
    return Operator(s)


def _same(a, b):
    sa, sb = a.samples(), b.samples()
    for x, y in zip([*a.fields(), sa.ts, sa.values, sa.energy], [*b.fields(), sb.ts, sb.values, sb.energy]):
        assert x.tobytes() == y.tobytes()


@pytest.mark.parametrize("n,wall,graded", [
    ((3, 3, 3), BC_PEC, False), ((2, 9, 40), BC_PEC, False), ((6, 35, 2), BC_PMC, False),
    ((33, 9, 65), BC_PMC, False), ((34, 33, 97), BC_PEC, True), ((20, 21, 22), BC_PML, False),
    ((41, 33, 64), BC_PML, False), ((30, 29, 35), BC_PML, True), ((104, 100, 98), BC_PEC, False)])
def test_resident_equals_direct(n, wall, graded):
    cop = CompressedOperator(_op(n, wall, graded))
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
