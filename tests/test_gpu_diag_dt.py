"""The time step and speed that come with the diagnostics are those of the copy, while the copy
engine is busy with another solver's fields and short steps run on."""
import threading

import numpy as np
import pytest

from gpu_helpers import config

pytestmark = pytest.mark.gpu


def _frames(pkg, n, wait):
    s = pkg.Solver.create(n=n, dyeScale=1)
    try:
        s.configure(config(viscosity=1.0, hyperP=2, forceAmp=0.2, forceK=n / 8, forceWidth=3.0, cfl=0.5, dtMin=1e-7, dtMax=1.0))
        s.reset({"k0": 6, "amplitude": 4, "seed": 3, "dyePattern": "none"})
        s.encodePrime()
        read = []
        for _ in range(60):
            s.encodeStep(); s.encodeReduce()
            s.encodeDiagnostics(); s.copyDiagnostics()
            if wait:
                s.synchronize()
            for _ in range(5):
                s.encodeStep(); s.encodeReduce()
            d = s.readDiagnostics()
            read.append((d["dt"], d["maxSpeed"], d["zonal"]))
        return read
    finally:
        s.destroy()


@pytest.mark.parametrize("n", [64, 256])
def test_the_time_step_read_is_that_of_the_copy(pkg, n):
    want = _frames(pkg, n, True)
    assert len({dt for dt, _, _ in want}) > 30      # the step size changes from frame to frame
    other = pkg.Solver.create(n=2048, dyeScale=1)
    stop = threading.Event()

    def read():
        while not stop.is_set():
            other.getBuffer("state0")
    t = threading.Thread(target=read)
    t.start()
    try:
        got = _frames(pkg, n, False)
    finally:
        stop.set()
        t.join()
        other.destroy()
    for (da, sa, za), (db, sb, zb) in zip(want, got):
        assert da == db and sa == sb and np.array_equal(za, zb)
