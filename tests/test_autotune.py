"""The autotuner's candidates, on the CPU (an engine that only records them)."""
import pytest

from wipems_gb300 import _abi, autotune, fdtd


@pytest.mark.parametrize("kernels", [("tma",), ("auto",), ("fused", "direct"), ()])
def test_candidates(monkeypatch, kernels):
    """The engine's own choice once, and every combination that was asked for."""
    made = []

    class Fake:
        def __init__(self, cop, device, stages, x_chunk, max_timesteps, kernel, tile_y):
            if kernel == "fused":
                raise _abi.FdtdError(1, "fdtd_engine_create", "not this grid")
            self.key = (kernel, tile_y, stages, x_chunk)
            made.append(self.key)

        def iterate(self, n):
            pass

        reset = close = lambda self: None

        def last_timing(self):
            return 1.0 + made.index(self.key), 1

        def stats(self):
            return dict(tile_y=self.key[1] or 4)

    monkeypatch.setattr(fdtd, "Engine", Fake)
    best, table = autotune.tune(object(), stages=(3, 4), xchunks=(1, 2), tile_ys=(4, 8), kernels=kernels)
    assert best["kernel"] == "auto" and best["stages"] == best["x_chunk"] == best["tile_y"] == 0
    want = {("auto", 0, 0, 0)}
    for k in kernels:
        if k != "fused":
            want |= {(k, ty, s, xc) for ty in ((4, 8) if k == "tma" else (0,)) for s in (3, 4) for xc in (1, 2)}
    assert set(made) == want and len(made) == len(want) == len(table)
