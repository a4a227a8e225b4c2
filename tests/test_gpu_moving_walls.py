"""Walls that move: a boundary particle's velocities come with its records, and nothing advances them. The project-U
force takes the approach viscosity and the XSPH term against a wall from its veleval, the other forces from its vel:
a step against the FP32 oracle, and a project-U step against the same passes called one by one, with eight, four and
two lanes a particle and with particles from the queue. Both sides add the same terms in another order: equal to 1e-5
of the largest value, as in the other parity tests."""
import numpy as np
import pytest

import sphmp
from helpers import device_ctx, download_state, field_err, in_grid_fluid, oracle_state
from oracle import oracle as O
from sphmp import abi, scenes
from test_gpu_lists import _cluster
from test_gpu_step_records import _by_calls

pytestmark = pytest.mark.gpu

RTOL = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _scene(kind, seed):
    """A scene whose boundary particles have a vel and another veleval, of the fluid's size."""
    if kind == "cluster":
        sc = _cluster(24, 9, seed)  # over two hundred neighbours, boundary particles among the fluid
    else:
        sc = scenes.small_block(seed=seed, n=kind, nphase=3, eos=abi.EOS_TAIT, velocity_scale=0.4,
                                dens=(1000.0, 800.0, 900.0), phase_frac=0.5)
    sc.params.mf_omega, sc.params.mf_visc_factor = 0.7, 1.3
    rng = np.random.default_rng(seed)
    wall = sc.disp["type"] == abi.TYPE_BOUNDARY
    for k in ("vel", "veleval"):
        sc.calc[k][wall] = rng.normal(0.0, 0.4, (int(wall.sum()), 3)).astype(np.float32)
    fluid = ~wall
    sc.calc["veleval"][fluid] = rng.normal(0.0, 0.4, (int(fluid.sum()), 3)).astype(np.float32)
    return sc


@pytest.mark.parametrize("schedule", [abi.SCHEDULE_FUSED, abi.SCHEDULE_REFERENCE, abi.SCHEDULE_PROJECTU])
@pytest.mark.parametrize("kind", [(14, 12, 13), "cluster"])
def test_step_matches_the_oracle(kind, schedule):
    sc = _scene(kind, 31)
    s = oracle_state(sc)
    O.before_first_step(sc.params, s)
    O.step(sc.params, s, schedule, 1)
    with device_ctx(sc) as ctx:
        ctx.before_first_step()
        ctx.step(1, schedule)
        ctx.sync()
        g = download_state(ctx)
    assert np.array_equal(g["midsort"], s.midsort)
    f = in_grid_fluid(s)
    keys = ("accel", "vel", "velxcor") if schedule == abi.SCHEDULE_PROJECTU else ("accel", "vel")
    for k in keys:
        assert np.abs(getattr(s, k)[f]).max() > 0, k
        assert field_err(g[k][f], getattr(s, k)[f]) < RTOL, k


@pytest.mark.parametrize("kind", [(14, 12, 13), (30, 24, 32), (64, 40, 56), "cluster"])
def test_projectu_step_equals_calls(kind):
    got = []
    for stepped in (True, False):
        with device_ctx(_scene(kind, 32)) as ctx:
            ctx.before_first_step()
            if stepped:
                ctx.step(1, abi.SCHEDULE_PROJECTU, use_graph=False)
            else:
                _by_calls(ctx, abi.SCHEDULE_PROJECTU)
            ctx.sync()
            got.append({f: ctx.download_field(f) for f in (abi.F_ACCEL, abi.F_VELXCOR, abi.F_VEL, abi.F_MIDSORT)})
    a, b = got
    assert np.array_equal(a[abi.F_MIDSORT], b[abi.F_MIDSORT])
    for f in (abi.F_ACCEL, abi.F_VELXCOR, abi.F_VEL):
        assert field_err(a[f], b[f]) < RTOL, f
