"""Stochastic forcing switched on and off by configure() between graph-replayed runs: a captured
substep belongs to the forcing it was captured with."""
import numpy as np
import pytest

from gpu_helpers import config, current_state

pytestmark = pytest.mark.gpu


def _run(pkg, n, fft, graph):
    s = pkg.Solver.create(n=n, dyeScale=1, fft=fft)
    try:
        out = []
        s.reset({"k0": 6, "amplitude": 3, "seed": 5, "dyePattern": "none"})
        for amp in (0.0, 0.2, 0.0):
            s.configure(config(viscosity=1.0, hyperP=2, forceAmp=amp, forceK=n / 8, forceWidth=3.0, dtMin=1e-3, dtMax=1e-3))
            s.step(12, dye=False, graph=graph, relatch=True)   # the same phase, dt slot and dye texture each time
            out.append(current_state(s))
        return out
    finally:
        s.destroy()


@pytest.mark.parametrize("n,fft", [(64, "fp32"), (256, "fp32"), (1024, "fp32"), (256, "tc-f16"), (1024, "tc-f16")])
def test_graphs_follow_the_forcing(pkg, n, fft):
    want, got = _run(pkg, n, fft, False), _run(pkg, n, fft, True)
    assert not np.array_equal(want[0], want[1])
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
