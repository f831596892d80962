"""Graphs of six substeps of the tensor-core solvers, their dye on a branch, against the same
substeps launched one by one: the same bits.  Every stage of the unfused steps writes the velocity
that the dye of the substep before reads."""
import numpy as np
import pytest

from gpu_helpers import config, current_state

pytestmark = pytest.mark.gpu


def _run(pkg, n, scale, fft, graph):
    s = pkg.Solver.create(n=n, dyeScale=scale, fft=fft)
    try:
        s.configure(config(viscosity=1.0, hyperP=2, forceAmp=0.1, forceK=n / 8, forceWidth=2.0, cfl=0.5, dtMax=2e-3))
        s.reset({"k0": 6, "amplitude": 4, "seed": 3, "dyePattern": "bands"})
        for steps in (7, 18, 6):
            s.step(steps, graph=graph, relatch=True)
        return current_state(s), s.currentDye, s.getBuffer("vel"), s.getBuffer("dt")[:2]
    finally:
        s.destroy()


@pytest.mark.parametrize("n,scale", [(256, 1), (256, 2), (256, 4), (512, 1), (512, 2), (1024, 1)])
@pytest.mark.parametrize("fft", ["tc-f16", "tc-bf16"])
def test_graphs_of_tensor_core_substeps_give_the_bits_of_single_launches(pkg, n, scale, fft):
    want, got = _run(pkg, n, scale, fft, False), _run(pkg, n, scale, fft, True)
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
