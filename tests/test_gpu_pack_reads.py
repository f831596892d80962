"""Calls that read the packs between two steps leave the run as it was: at 4096^2 the pair kernels
keep the packs in blocks of four columns, below that in rows, and a step after such a call takes
neither for the other."""
import numpy as np
import pytest

from gpu_helpers import config, current_state

pytestmark = pytest.mark.gpu

READS = {"packA": lambda s: s.getBuffer("packA"), "packB": lambda s: s.getBuffer("packB"),
         "both": lambda s: (s.getBuffer("packA"), s.getBuffer("packB")), "nlPack": lambda s: s.nlPack()}


def _run(pkg, n, graph, read):
    s = pkg.Solver.create(n=n, dyeScale=1)
    try:
        s.configure(config(beta=7.0, drag=1e-2, viscosity=1.0, hyperP=2, cfl=0.5, dtMax=1e-3))
        s.reset({"k0": 6, "amplitude": 3, "seed": 5, "dyePattern": "none"})
        for _ in range(2):
            s.step(2, dye=False, graph=graph)
            if read:
                READS[read](s)
        s.encodeStep()
        return current_state(s), s.getBuffer("vel"), s.getBuffer("dt")[:2]
    finally:
        s.destroy()


@pytest.mark.parametrize("n", [128, 1024, 4096])
@pytest.mark.parametrize("graph", [False, True])
def test_a_read_of_the_packs_leaves_the_next_step_alone(pkg, n, graph):
    """The packs are made again from the state where the read undid their layout: the same kernel
    forms them from the same values, so the bits are those of the run that read nothing."""
    want = _run(pkg, n, graph, None)
    assert np.all(np.isfinite(want[0].view(np.float32))) and np.any(want[0])
    for read in READS:
        got = _run(pkg, n, graph, read)
        for a, b in zip(want, got):
            assert np.array_equal(a, b), read


def test_a_second_read_returns_the_first(pkg):
    s = pkg.Solver.create(n=4096, dyeScale=1)
    try:
        s.configure(config(viscosity=1.0, hyperP=2, dtMax=1e-3))
        s.reset({"k0": 6, "amplitude": 3, "seed": 5, "dyePattern": "none"})
        s.step(1, dye=False)
        first = [s.getBuffer("packA"), s.getBuffer("packB")]
        again = [s.getBuffer("packA"), s.getBuffer("packB")]
        assert all(np.array_equal(a, b) for a, b in zip(first, again))
        assert np.array_equal(first[1][1], np.conj(first[1][-1])) and np.any(first[1][1])
    finally:
        s.destroy()


@pytest.mark.parametrize("n", [1024, 4096])
def test_packs_of_an_earlier_state_are_kept(pkg, n):
    """The packs as the last step left them, read at once and after the state they belong to has been
    replaced: the same bits, whichever way the read puts them in rows."""
    out = []
    for stale in (False, True):
        s = pkg.Solver.create(n=n, dyeScale=1)
        try:
            s.configure(config(viscosity=1.0, hyperP=2, dtMax=1e-3))
            s.reset({"k0": 6, "amplitude": 3, "seed": 5, "dyePattern": "none"})
            s.step(2, dye=False)
            if stale:
                s.setBuffer("state%d" % s.phase, np.zeros((n, n), np.complex64))
            out.append([s.getBuffer("packA"), s.getBuffer("packB")])
        finally:
            s.destroy()
    assert np.any(out[0][0]) and np.any(out[0][1])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
