"""Long graph-replayed runs (graphs of six substeps, the dye of small textures on a branch beside
the next substep) against the same substeps launched one by one: the same bits, also across
changes of splats and flags and with diagnostics in between."""
import numpy as np
import pytest

from gpu_helpers import config, current_state

pytestmark = pytest.mark.gpu

SPLAT = {"x": 0.3, "y": 0.6, "dx": 0.004, "dy": -0.002, "color": (1.0, 0.5, 0.2), "radius": 0.06, "amp": 50.0,
         "dyeAmp": 0.5}


def _run(pkg, n, scale, graph, relatch):
    s = pkg.Solver.create(n=n, dyeScale=scale)
    try:
        s.configure(config(viscosity=1.0, hyperP=2, forceAmp=0.1, forceK=n / 8, forceWidth=2.0, cfl=0.5, dtMax=2e-3))
        s.reset({"k0": 6, "amplitude": 4, "seed": 3, "dyePattern": "bands"})
        s.step(13, graph=graph, relatch=relatch)
        s.setSplats([SPLAT])
        s.step(7, graph=graph, relatch=relatch)
        s.encodeDiagnostics()
        s.copyDiagnostics()
        s.step(6, dye=False, graph=graph, relatch=relatch)
        s.setSplats([])
        s.step(12, reduce=False, graph=graph, relatch=relatch)
        s.step(25, graph=graph, relatch=relatch)
        d = s.readDiagnostics()
        return [current_state(s), s.currentDye, s.getBuffer("vel"), s.getBuffer("dt")[:2], d["spectrum"], d["zonal"],
                np.array([s.phase, s.dyeParity, s.stepIndex])]
    finally:
        s.destroy()


@pytest.mark.parametrize("n,scale", [(32, 2), (64, 4), (128, 1), (256, 2), (512, 2), (1024, 1), (1024, 2)])
@pytest.mark.parametrize("relatch", [False, True])
def test_graphs_of_substeps_give_the_bits_of_single_launches(pkg, n, scale, relatch):
    want, got = _run(pkg, n, scale, False, relatch), _run(pkg, n, scale, True, relatch)
    for i, (a, b) in enumerate(zip(want, got)):
        if i == 4:      # FP64 sums by atomics: any order
            assert np.allclose(a, b, rtol=1e-12, atol=0)
        else:
            assert np.array_equal(a, b), i


@pytest.mark.parametrize("n,scale", [(64, 2), (256, 2), (512, 1)])
def test_single_encodes_run_beside_the_spectra(pkg, n, scale):
    """A frame loop of single encode calls, its diagnostics read a frame late, against the same
    calls each waited for: the step behind the diagnostics may run beside the spectra, the one
    after it writes the state that they read."""
    out = []
    for wait in (True, False):
        s = pkg.Solver.create(n=n, dyeScale=scale)
        try:
            s.configure(config(viscosity=1.0, hyperP=2, forceAmp=0.1, forceK=n / 8, forceWidth=2.0, cfl=0.5, dtMax=2e-3))
            s.reset({"k0": 6, "amplitude": 4, "seed": 3, "dyePattern": "bands"})
            s.encodePrime()
            calls, read = [], []
            for frame in range(12):
                calls = [s.encodeStep, s.encodeDye, s.encodeReduce] * (frame % 3 + 1) + [s.encodeDiagnostics]
                if frame % 4 == 3:
                    calls += [s.encodeDiagnostics]
                for call in calls:
                    call()
                    if wait:
                        s.synchronize()
                read.append(s.readDiagnostics())
                s.copyDiagnostics()
                if wait:
                    s.synchronize()
            read.append(s.readDiagnostics())
            out.append(([r for r in read if r], current_state(s), s.currentDye, s.readDiagnosticsFixed()))
        finally:
            s.destroy()
    (ra, sa, da, fa), (rb, sb, db, fb) = out
    assert np.array_equal(sa, sb) and np.array_equal(da, db) and len(ra) == len(rb) == 12
    for a, b in zip(ra, rb):
        assert np.allclose(a["spectrum"], b["spectrum"], rtol=1e-12, atol=0)
        assert np.array_equal(a["zonal"], b["zonal"]) and a["dt"] == b["dt"] and a["maxSpeed"] == b["maxSpeed"]
    assert np.array_equal(fa["spectrum"], fb["spectrum"])
