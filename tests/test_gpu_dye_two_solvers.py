"""Two solvers whose dye kernels share a tile shape but not its window sizes: making the second
leaves the first able to run, whichever comes first."""
import numpy as np
import pytest

from gpu_helpers import config

pytestmark = pytest.mark.gpu


def _solver(pkg, n, scale):
    s = pkg.Solver.create(n=n, dyeScale=scale)
    s.configure(config(viscosity=1.0, hyperP=2, dtMax=1e-3))
    s.reset({"k0": 6, "amplitude": 3, "seed": 5, "dyePattern": "bands"})
    return s


@pytest.mark.parametrize("a,b", [((256, 1), (128, 2)), ((256, 1), (64, 4)), ((1024, 2), (512, 4)), ((512, 2), (256, 4))])
def test_the_larger_windows_still_launch(pkg, a, b):
    alone = _solver(pkg, *a)
    try:
        alone.step(2)
        want = alone.currentDye
    finally:
        alone.destroy()
    one = _solver(pkg, *a)
    two = _solver(pkg, *b)
    try:
        two.step(1)
        one.step(2)
        assert np.array_equal(one.currentDye, want)
    finally:
        one.destroy()
        two.destroy()
