"""The residue of an IISPH solve, which its tolerance is compared with, against the oracle in 64 bits. It is a mean over
the particles of what is left of sums as large as the first iteration's residue: rounding errors that differ from
particle to particle average out, so what remains is bounded by an error of one sign, which is asked to stay below
half of one rounding (2^-25) of those sums, at every iteration. The walls' volumes are the device's on both sides."""
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


@pytest.mark.parametrize("n,h,walls", [((32, 32, 32), 0.02, True), ((30, 34, 31), 0.02, False), ((33, 30, 32), 0.0125, True)])
def test_residue_against_64_bits(n, h, walls):
    d = h / 2
    box = tuple(k * d * f for k, f in zip(n, (2.0, 1.5, 1.25)))
    sc = scenes.small_block(seed=7, n=n, d=d, h=h, box=box, dt=1e-2 * h, nphase=1, eos=abi.EOS_TAIT, dens=(1000.0,),
                            multiphase=0, walls=walls)
    p, s = sc.params, oracle_state(sc, np.float64)
    O.before_first_step(p, s)
    with device_ctx(sc) as ctx:
        ctx.before_first_step()
        g = download_state(ctx)
        assert np.array_equal(g["bornid"], s.bornid) and np.array_equal(g["midsort"], s.midsort)
        wall = s.type == abi.TYPE_BOUNDARY
        s.dens[wall] = g["dens"][wall]
        fluid = in_grid_fluid(s)
        O.call("orc_iisph_density", p, s)
        O.call("orc_iisph_predict", p, s)
        ctx.iisph_density()
        ctx.iisph_predict_advection()
        for it in range(10):
            want = O.call("orc_iisph_iteration", p, s)
            got = ctx.iisph_pressure_iteration()
            mean = float(np.abs(s.residue[fluid]).mean())
            first = abs(want) if it == 0 else first
            first_mean = mean if it == 0 else first_mean
            assert abs(got[0] - want) < 2.0 ** -25 * first, it
            assert abs(got[1] - mean) < 2.0 ** -23 * first_mean, it
