"""Densities against the oracle in 64 bits. The terms of a sum round differently, and so do the particles' sums, so their
mean error is that of what is common to all: asked to stay below a quarter of one rounding (2^-26), for radii whose
square rounds up, down and hardly at all, by the bucket kernel with few and many members a bucket and by the search of
the cells. The walls' volumes are the device's on both sides."""
import numpy as np
import pytest

import sphmp
from helpers import device_ctx, download_state, in_grid_fluid, oracle_state
from oracle import oracle as O
from sphmp import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


@pytest.mark.parametrize("search", [False, True])
@pytest.mark.parametrize("h,scale,per", [(0.02, 1.0, 2.0), (0.0125, 1.0, 2.0), (0.03, 1.0, 2.0), (0.015625, 1.0, 2.0), (0.011, 0.5, 2.0),
                                         (0.02, 1.0, 3.1)])
def test_mean_error_of_the_density(h, scale, per, search):
    sc = scenes.small_block(seed=12, n=(40, 40, 40), d=h / per / scale, h=h, simscale=scale, nphase=1, dens=(1000.0,),
                            eos=abi.EOS_LINEAR)
    p, s = sc.params, oracle_state(sc, np.float64)
    O.before_first_step(p, s)
    with device_ctx(sc) as ctx:
        ctx.before_first_step()
        ctx.sort()
        if search:  # positions put in after the sort (the same ones)
            ctx.upload_field(abi.F_POS, ctx.download_field(abi.F_POS))
        g = download_state(ctx)
        wall = s.type == abi.TYPE_BOUNDARY
        assert np.array_equal(g["bornid"], s.bornid) and np.array_equal(g["type"], s.type)
        s.dens[wall] = g["dens"][wall]
        O.call("orc_compute_pressure", p, s)
        ctx.compute_pressure()
        g = download_state(ctx)
    f = in_grid_fluid(s)
    assert f.sum() > 60000
    assert abs(float(np.mean(g["dens"][f] / s.dens[f] - 1.0))) < 2.0 ** -26
