"""Steps that a caller captures into a graph of its own, replayed after a state of another kind has
been stored: the graph was captured when the state was dealiased, the stored one has cells outside
the 2/3 band."""
import numpy as np
import pytest

from conftest import rel_l2
from gpu_helpers import config, current_state, set_fixed_dt

pytestmark = pytest.mark.gpu

# as between the two kinds of stage kernels: FP32 transforms in another order, three stages a step
TOL = 2e-6


def _fields(n):
    rng = np.random.default_rng(n)
    raw = np.fft.fft2(rng.standard_normal((n, n))).astype(np.complex64)
    raw[0, 0] = 0
    k = np.abs(np.fft.fftfreq(n, 1.0 / n))
    return raw, raw * ((k[:, None] < n / 3.0) & (k[None, :] < n / 3.0))


@pytest.mark.parametrize("n", [64, 256])
def test_a_captured_solver_step_takes_any_state(pkg, n):
    import torch
    raw, band = _fields(n)
    s = pkg.Solver.create(n=n, dyeScale=1)
    try:
        s.configure(config(beta=3.0, drag=1e-2, viscosity=1.0, hyperP=1))
        s.setSplats([])
        set_fixed_dt(s, 1e-3)
        want = []
        for w in (band, raw):
            s.phase = 0
            s.setBuffer("state0", w)
            for _ in range(3):
                s.encodeStep()
            want.append(current_state(s))
        s.reset({"amplitude": 0, "dyePattern": "none"})   # dealiased states again
        set_fixed_dt(s, 1e-3)
        s.setBuffer("state0", band)
        s.synchronize()
        st = torch.cuda.ExternalStream(s.stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            for _ in range(3):
                s.encodeStep()
        assert s.phase == 0
        for w, ref in zip((band, raw), want):
            s.setBuffer("state0", w)
            with torch.cuda.stream(st):
                g.replay()
            torch.cuda.synchronize()
            assert rel_l2(s.getBuffer("state0"), ref) <= TOL
        del g
    finally:
        s.destroy()


@pytest.mark.parametrize("n", [64, 256])
@pytest.mark.parametrize("graph", [False, True])
def test_captured_steps_and_direct_ones_in_turn(pkg, n, graph):
    """Replays and direct runs of three steps each, the state going from one to the other."""
    import torch
    band = _fields(n)[1]
    out = []
    for captured in (False, True):
        s = pkg.Solver.create(n=n, dyeScale=1)
        try:
            # one step size in both dt slots: step() primes, which takes the other slot
            s.configure(config(beta=3.0, drag=1e-2, viscosity=1.0, hyperP=1, dtMin=1e-3, dtMax=1e-3))
            s.setSplats([])
            set_fixed_dt(s, 1e-3)
            s.setBuffer("state0", band)
            s.encodeStep()
            s.phase = 0                      # the packs are laid out for the pair kernels
            s.setBuffer("state0", band)
            s.synchronize()
            if captured:
                st = torch.cuda.ExternalStream(s.stream)
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=st):
                    for _ in range(3):
                        s.encodeStep()
            for _ in range(3):
                if captured:
                    with torch.cuda.stream(st):
                        g.replay()
                else:
                    for _ in range(3):
                        s.encodeStep()
                s.step(3, dye=False, reduce=False, graph=graph)
            out.append(current_state(s))
            if captured:
                del g
        finally:
            s.destroy()
    # nine such steps on each side; the first ones' difference is carried on, not amplified, by dt |N| / |w| << 1
    assert rel_l2(out[1], out[0]) <= 6 * TOL
    assert np.any(out[0])


@pytest.mark.parametrize("n", [64])
def test_a_captured_prime_takes_any_state(pkg, n):
    import torch
    raw, band = _fields(n)
    s = pkg.Solver.create(n=n, dyeScale=1)
    try:
        s.configure(config(viscosity=1.0, hyperP=1))
        s.setBuffer("state0", raw)
        s.encodePrime()
        want = s.getBuffer("vel")
        s.reset({"amplitude": 0, "dyePattern": "none"})
        s.setBuffer("state0", band)
        s.synchronize()
        st = torch.cuda.ExternalStream(s.stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            s.encodePrime()
        s.setBuffer("state0", raw)
        with torch.cuda.stream(st):
            g.replay()
        torch.cuda.synchronize()
        assert rel_l2(s.getBuffer("vel"), want) <= TOL
        del g
    finally:
        s.destroy()


def test_a_captured_ensemble_step_takes_any_state(pkg):
    import torch
    sizes = [64, 128]
    e = pkg.Ensemble([{"n": n, "beta": 2.0, "drag": 1e-2, "nuH": 1e-4, "hyperP": 1, "dt": 1e-3} for n in sizes])
    try:
        fields = [_fields(n) for n in sizes]

        def store(kind):
            for i, f in enumerate(fields):
                e.setState(i, f[kind])

        def read():
            return [e.getState(i) for i in range(len(sizes))]
        want = []
        for kind in (1, 0):
            store(kind)
            e.step(3, graph=False)
            want.append(read())
        e.seedBand(4.0, 12.0, 1.0)      # dealiased states again
        store(1)
        e.synchronize()
        st = torch.cuda.ExternalStream(e.stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            e.step(3, graph=False)
        for kind, ref in zip((1, 0), want):
            store(kind)
            with torch.cuda.stream(st):
                g.replay()
            torch.cuda.synchronize()
            for a, b in zip(read(), ref):
                assert rel_l2(a, b) <= TOL
        del g
    finally:
        e.destroy()
