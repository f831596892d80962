"""The fused dye step against the reference's three dispatches, bit for bit, over its tile shapes
and the two kinds of tile whose traces stay under a texel: inside the texture (positions never
wrap) and on its edge."""
import numpy as np
import pytest

from gpu_helpers import config, set_fixed_dt

pytestmark = pytest.mark.gpu


def _texture(m, seed, special):
    rng = np.random.default_rng(seed)
    t = rng.uniform(-1.0, 1.0, (m, m, 4)).astype(np.float16)
    t[rng.random((m, m, 4)) < 0.1] = np.float16(-0.0)
    t[rng.random((m, m, 4)) < 0.05] = np.float16(6e-8)        # subnormal
    t[rng.random((m, m, 4)) < 0.02] = np.float16(65504.0)
    if special:
        t[rng.random((m, m, 4)) < 0.003] = np.float16(np.inf)
        t[rng.random((m, m, 4)) < 0.003] = np.float16(np.nan)
    return t.view(np.uint16)


# (grid, dye scale): 32 x 8 tiles up to 256 texels, 32 x 32 on an unrefined dye, 64 x 32 above
@pytest.mark.parametrize("n,scale", [(32, 1), (32, 4), (64, 2), (128, 2), (256, 1), (512, 1), (256, 2), (128, 4), (512, 2)])
@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("splat", [False, True])
def test_tiles_match_the_three_passes(pkg, n, scale, special, splat):
    s = pkg.Solver.create(n=n, dyeScale=scale)
    try:
        s.configure(config(viscosity=1.0, cfl=0.5, dtMax=0.02, dyeFade=0.97))
        s.reset({"k0": n / 10, "amplitude": 10, "seed": n, "dyePattern": "none"})
        s.setSplats([{"x": 0.5, "y": 0.01, "dx": 0.0, "dy": 0.0, "color": (0.4, -0.3, 0.7), "radius": 0.2,
                      "amp": 0.0, "dyeAmp": 1.0}] if splat else [])
        s.encodePrime()
        vel = s.getBuffer("vel")
        top = float(max(np.abs(vel.real).max(), np.abs(vel.imag).max()))
        start = _texture(n * scale, 7 * n + scale, special)
        for texels in (0.9, 0.2):
            set_fixed_dt(s, texels * 2 * np.pi / (top * n * scale))
            got = []
            for step in (s.encodeDye, s.encodeDyePasses):
                s.dyeParity = 0
                s.setDye(start)
                step()
                got.append(s.currentDye)
            a, b = got
            nan = [np.isnan(x.view(np.float16)) for x in got]
            assert np.array_equal(nan[0], nan[1])
            assert np.array_equal(a[~nan[0]], b[~nan[1]])
    finally:
        s.destroy()
