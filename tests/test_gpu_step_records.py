"""The alpha advance and the project-U force of a step read the neighbour records that the step's drift pass wrote,
with eight, four, two or one lane a particle and the particles with many neighbours from a queue; called one by one,
the passes gather the fields themselves with one thread a particle. Both add the same terms in another order: equal to
1e-5 of the largest value, as in the other parity tests (sums of at most a few hundred FP32 terms)."""
import numpy as np
import pytest

import sphmp
from helpers import device_ctx, field_err
from sphmp import abi, scenes
from test_gpu_lists import _cluster

pytestmark = pytest.mark.gpu

RTOL = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _by_calls(ctx, schedule):
    ctx.sort()
    ctx.compute_pressure()
    ctx.compute_drift_vel()
    ctx.compute_alpha_advance()
    ctx.compute_correction()
    if schedule == abi.SCHEDULE_PROJECTU:
        ctx.compute_force_projectu()
    else:
        ctx.compute_force()
    ctx.advance()


def _scene(lattice, nphase):
    if lattice == "cluster":
        sc = _cluster(24, 9, 400)  # over two hundred neighbours
    else:
        d = 0.005
        sc = scenes.blobs_3phase(seed=9, lattice=lattice, box=(2 * lattice[0] * d, 2 * lattice[1] * d, lattice[2] * d),
                                 n_blobs=16)
    if nphase < 3:  # the particles of the dropped phases join the first
        sc.params.nphase = nphase
        kept = [sc.params.densArr[k] for k in range(nphase)]
        sc.calc["restdens"][~np.isin(sc.calc["restdens"], np.float32(kept))] = kept[0]
    return sc


@pytest.mark.parametrize("schedule", [abi.SCHEDULE_REFERENCE, abi.SCHEDULE_PROJECTU])
@pytest.mark.parametrize("lattice,nphase", [((24, 16, 24), 3), ((30, 24, 32), 2), ((60, 40, 60), 3), ((96, 64, 80), 2),
                                            ("cluster", 3), ("cluster", 1)])
def test_step_equals_calls(schedule, lattice, nphase):
    sc = _scene(lattice, nphase)
    got = []
    for stepped in (True, False):
        ctx = device_ctx(sc)
        ctx.before_first_step()
        ctx.step(1, abi.SCHEDULE_FUSED)  # drift velocities and fractions that differ between particles
        if stepped:
            ctx.step(1, schedule, use_graph=False)
        else:
            _by_calls(ctx, schedule)
        ctx.sync()
        got.append({f: ctx.download_field(f) for f in (abi.F_ALPHA, abi.F_ACCEL, abi.F_VELXCOR, abi.F_VEL, abi.F_MIDSORT)})
        ctx.close()
    a, b = got
    assert np.array_equal(a[abi.F_MIDSORT], b[abi.F_MIDSORT])
    for f in (abi.F_ALPHA, abi.F_ACCEL, abi.F_VEL):
        assert field_err(a[f], b[f], floor=1.0 if f == abi.F_ALPHA else 0.0) < RTOL, f
    if schedule == abi.SCHEDULE_PROJECTU:
        assert field_err(a[abi.F_VELXCOR], b[abi.F_VELXCOR]) < RTOL
