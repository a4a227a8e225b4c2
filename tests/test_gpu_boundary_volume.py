"""Boundary volumes 1 / (kpoly6 sum (h^2 - r^2)^3) against numpy in 64 bits. Every term carries its rounding errors and
the sum too, so the volume is the exact one rounded once: half a unit in the last place (2^-24 of the value at most),
and 2e-8 for what is left before that rounding (differences of positions are exact but where a coordinate changes sign,
there up to 2^-24 of the difference)."""
import numpy as np
import pytest

import sphmp
from helpers import device_ctx
from sphmp import abi, scenes
from test_gpu_lists import _cluster

pytestmark = pytest.mark.gpu

BOUND = 2.0 ** -24 + 2e-8


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _exact(p, pos):
    x = pos.astype(np.float64) * float(p.simscale)
    h2 = float(p.smoothradius) ** 2
    v = np.empty(len(x))
    for i in range(0, len(x), 256):
        r2 = ((x[i:i + 256, None] - x[None]) ** 2).sum(2)
        v[i:i + 256] = 1.0 / (float(p.kpoly6) * (np.maximum(h2 - r2, 0.0) ** 3).sum(1))
    return v


def _scene(kind):
    if kind == "cluster":  # boundary particles at random
        return _cluster(40, 20, 3)
    if kind == "coincident":
        sc = _cluster(40, 20, 4)
        sc.disp["pos"][:] = sc.disp["pos"][0]
        return sc
    h, scale = kind
    return scenes.small_block(seed=2, n=(8, 8, 8), d=h / 2 / scale, h=h, simscale=scale, nphase=1, dens=(1000.0,))


@pytest.mark.parametrize("kind", [(0.02, 1.0), (0.0125, 1.0), (0.01, 0.5), (0.01, 0.004), (3.0, 1.0), (2e-3, 1.0),
                                  "cluster", "coincident"])
def test_volume_is_exact(kind):
    sc = _scene(kind)
    with device_ctx(sc) as ctx:
        ctx.before_first_step()
        wall = (ctx.download_field(abi.F_TYPE) == abi.TYPE_BOUNDARY) & (ctx.download_field(abi.F_MGCELL) != abi.GRID_UNDEF)
        pos, v = ctx.download_field(abi.F_POS)[wall], ctx.download_field(abi.F_DENS)[wall]
    assert wall.sum() > 50
    want = _exact(sc.params, pos)
    assert np.abs(v / want - 1.0).max() < BOUND
