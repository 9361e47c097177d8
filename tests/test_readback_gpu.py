"""Field readback and dumps on every device-axis rotation: the packed copies
(32 x 32 tiles turned over on the device) must equal single-node reads and
the unrotated engine bit for bit, at extents around the tile edges."""
import numpy as np
import pytest

from wipems_gb300 import CompressedOperator, Engine, Operator, Scene
from wipems_gb300.fdtd import BC_PEC

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("libs")]


def _op(n):
    s = Scene(*[np.arange(k, dtype=float) for k in n], 1e-3)
    s.set_boundary([BC_PEC] * 6)
    s.set_gauss_excite(20e9, 20e9, 200)
    c = [k // 2 for k in n]
    s.add_excitation(c, [c[0], c[1], c[2] + 1], [0.0, 0.0, 1.0])
    return Operator(s)


@pytest.mark.parametrize("n", [(3, 4, 5), (31, 33, 32), (64, 65, 34), (97, 6, 130)])
def test_rotated_readback(n):
    op = _op(n)
    rng = np.random.default_rng(3)
    nodes = [[int(rng.integers(0, k)) for k in n] for _ in range(20)] + [[0, 0, 0], [k - 1 for k in n]]
    ref = None
    for rot in (0, 1, 2):
        e = Engine(CompressedOperator(op, rotation=rot), kernel="tma")
        e.iterate(40)
        V, I = e.fields()
        assert np.any(V) and np.any(I)
        for x, y, z in nodes:
            for c in range(3):
                assert V[c, x, y, z] == e.get_volt(c, x, y, z) and I[c, x, y, z] == e.get_curr(c, x, y, z)
        out = [V, I, e.dump_field("E", "node"), e.dump_field("H", "cell", start=(0, 1, 1), step=(1, 2, 3)),
               e.dump_field("H", "node", step=(2, 1, 1))]
        e.close()
        if ref is None:
            ref = out
        for a, b in zip(ref, out):
            assert a.shape == b.shape and a.tobytes() == b.tobytes()
