"""The pair kernels (dealiased states, two lines per thread) against the stage kernels that take
any state, at every grid size: edges of the band, spare groups of the last CTA, every radix
tail; and the states the pair kernels must not take."""
import numpy as np
import pytest

from conftest import rel_l2
from gpu_helpers import config, current_state, load_state, set_fixed_dt

pytestmark = pytest.mark.gpu

# Both kernels evaluate the same formulas in FP32 with differently ordered transforms: each is
# within about eps sqrt(log2 N^2) ~ 3e-7 of the exact transforms per stage, and a step of dt
# scales the right-hand side's error by dt |N| / |w| < 1.  2e-6 leaves room for three stages
# and both sides.
TOL = 2e-6
SPLAT = {"x": 0.3, "y": 0.6, "dx": 0.004, "dy": -0.002, "color": (1.0, 0.5, 0.2), "radius": 0.06, "amp": 50.0,
         "dyeAmp": 0.5}


def _shapes(s):
    col = s.tuneVariantNames("column")
    row = s.tuneVariantNames("row")
    assert col[0] == "column pairs" and row[0] == "row pairs"
    return (0, 0), (1, 1), (1, 0), (0, 1)


def _stepped(s, n, shape, steps=2, splat=True):
    s.tuneSelect(*shape)
    s.configure(config(beta=7.0, drag=1e-2, viscosity=1.0, hyperP=2, forceAmp=0.1, forceK=n / 8, forceWidth=2.0,
                       cfl=0.5, dtMax=1e-3))
    s.reset({"k0": 6, "amplitude": 3, "seed": 5, "dyePattern": "none"})
    s.setSplats([SPLAT] if splat else [])
    s.step(steps, dye=False, reduce=True, graph=False, relatch=True)
    return {"state": current_state(s), "vel": s.getBuffer("vel"), "dt": s.getBuffer("dt")[:2],
            "packA": s.getBuffer("packA"), "packB": s.getBuffer("packB")}


@pytest.mark.parametrize("n", [32, 64, 128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("splat", [False, True])
def test_pair_kernels_match_the_any_state_kernels(pkg, n, splat):
    if splat and n > 1024:
        pytest.skip("pointer force is the same code at every size")
    s = pkg.Solver.create(n=n, dyeScale=1)
    try:
        pairs, general, mixed, fallback = _shapes(s)
        want = _stepped(s, n, general, splat=splat)
        for shape in (pairs, mixed, fallback):
            got = _stepped(s, n, shape, splat=splat)
            for key in want:
                assert rel_l2(got[key], want[key]) <= TOL, (shape, key, rel_l2(got[key], want[key]))
            ky = np.abs(np.fft.fftfreq(n, 1.0 / n))
            out = (ky[:, None] >= n / 3.0) | (ky[None, :] >= n / 3.0)
            assert not np.any(got["state"][out])
    finally:
        s.destroy()


@pytest.mark.parametrize("n", [32, 128, 256])
def test_states_that_are_not_hermitian_step_alike(pkg, n):
    """Complex noise inside the band, not Hermitian: the stage reads real parts of its inverse
    transforms whatever the state."""
    rng = np.random.default_rng(n)
    ky = np.abs(np.fft.fftfreq(n, 1.0 / n))
    band = (ky[:, None] < n / 3.0) & (ky[None, :] < n / 3.0)
    w = ((rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * band * n).astype(np.complex64)
    w[0, 0] = 0
    s = pkg.Solver.create(n=n, dyeScale=1)
    try:
        outs = []
        for shape in _shapes(s)[:3]:
            s.tuneSelect(*shape)
            s.configure(config(beta=3.0, drag=1e-2, viscosity=1.0, hyperP=1))
            load_state(s, w)
            set_fixed_dt(s, 1e-3)
            for _ in range(2):
                s.encodeStep()
            outs.append(current_state(s))
        assert rel_l2(outs[0], outs[1]) <= TOL and rel_l2(outs[2], outs[1]) <= TOL
    finally:
        s.destroy()


@pytest.mark.parametrize("graph", [False, True])
def test_cells_outside_the_band_take_the_any_state_kernels(pkg, graph):
    """A stored state with cells outside the band steps through the kernels that take any state
    (the same bits as with those selected), and a later reset returns to the pair kernels."""
    n = 64
    rng = np.random.default_rng(3)
    w = np.fft.fft2(rng.standard_normal((n, n))).astype(np.complex64)
    w[0, 0] = 0
    outs = []
    s = pkg.Solver.create(n=n, dyeScale=1)
    try:
        for shape in ((0, 0), (1, 1)):
            s.tuneSelect(*shape)
            s.configure(config(viscosity=0.5, hyperP=1, dtMin=1e-3, dtMax=1e-3))
            s.reset({"amplitude": 0, "dyePattern": "none"})
            s.step(2, dye=False, graph=graph)          # graphs of a dealiased state exist
            load_state(s, w)
            s.step(3, dye=False, graph=graph)
            outs.append(current_state(s))
        assert np.array_equal(*outs)
        assert np.any(outs[0][n // 2])
        s.tuneSelect(0, 0)
        a = _stepped(s, n, (0, 0))["state"]
    finally:
        s.destroy()
    fresh = pkg.Solver.create(n=n, dyeScale=1)
    try:
        assert np.array_equal(a, _stepped(fresh, n, (0, 0))["state"])
    finally:
        fresh.destroy()


@pytest.mark.parametrize("banded", [True, False])
def test_ensemble_states(pkg, banded):
    """Every ensemble size, work lists with spare groups, through the default shapes and the
    any-state ones; a member outside the band moves the whole batch to the latter."""
    sizes = [64, 64, 64, 128, 256, 512, 1024]
    inst = [{"n": n, "beta": 2.0 * k, "drag": 1e-2, "nuH": 1e-4, "hyperP": 1, "dt": 1e-3, "seed": k, "forceAmp": 0.05,
             "forceK": n / 8, "forceWidth": 2.0} for k, n in enumerate(sizes)]
    e = pkg.Ensemble(inst)
    try:
        outs = []
        for shape in ((0, 0), (1, 1), (1, 0), (0, 1)):
            e.tuneSelect(*shape)
            e.seedBand(4.0, 12.0, 1.0)
            if not banded:
                w = e.getState(1)
                w[32, 5] = 64.0
                e.setState(1, w)
            e.step(4)
            outs.append([e.getState(i) for i in range(len(sizes))])
        for got in outs[1:]:
            for a, b in zip(got, outs[1]):
                assert rel_l2(a, b) <= TOL
        for a, b in zip(outs[0], outs[1]):
            assert rel_l2(a, b) <= TOL
            assert banded or np.array_equal(a, b)
    finally:
        e.destroy()


@pytest.mark.parametrize("n", [32, 64, 128])
@pytest.mark.parametrize("splat", [False, True])
def test_the_step_in_one_launch_matches_its_stages(pkg, n, splat):
    """The small grids' one-launch step against the same step launched stage by stage (as the
    profiler times it): state ring, velocity, dt and packs."""
    outs = []
    for apart in (False, True):
        s = pkg.Solver.create(n=n, dyeScale=1)
        try:
            s.profile(apart)
            outs.append(_stepped(s, n, (0, 0), steps=4, splat=splat))
            outs[-1]["ring"] = np.stack([s.getBuffer(f"state{i}") for i in range(3)])
        finally:
            s.destroy()
    for key in outs[0]:
        assert rel_l2(outs[0][key], outs[1][key]) <= TOL, key
