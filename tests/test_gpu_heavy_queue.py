"""The queue of particles with many neighbours belongs to the lists of one density pass. A density pass over cells
that do not match the positions any more queues nobody, and a context that took over another's state has no lists:
the forces are then those of a context that never had a queue, bit for bit (the same sums in the same order)."""
import numpy as np
import pytest

import sphmp
from helpers import bits_equal, device_ctx
from sphmp import abi, scenes
from test_gpu_sort_calls import _dense

pytestmark = pytest.mark.gpu

FIELDS = (abi.F_POS, abi.F_DENS, abi.F_PRESSURE, abi.F_ACCEL)


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _moved_forces(ctx, shift):
    """Density and forces at positions uploaded without a sort."""
    pos = ctx.download_field(abi.F_POS)
    ctx.upload_field(abi.F_POS, pos + shift)
    ctx.compute_pressure()
    ctx.compute_force()
    return [ctx.download_field(f) for f in FIELDS]


def _shift(n, size):
    return np.random.default_rng(n).uniform(-size, size, (n, 3)).astype(np.float32)


def test_density_without_a_sort_queues_nobody():
    sc = _dense(40)  # about 170 neighbours, more than the queue's threshold
    got = []
    for queued in (False, True):
        with device_ctx(sc) as ctx:
            ctx.before_first_step()
            ctx.sort()
            if queued:
                ctx.compute_pressure()
            got.append(_moved_forces(ctx, _shift(sc.n, 1e-4)))
    assert np.abs(got[0][-1]).max() > 0
    for f, a, b in zip(FIELDS, *got):
        assert bits_equal(a, b), f


def test_state_taken_over_by_a_fallback():
    sc = scenes.rollout_bubbles(seed=4, lattice=(16, 16, 16), liquid_only=True)
    sc.params.heavy_list = 32  # most of the particles
    with device_ctx(sc) as ctx, sphmp.Context(sc.params) as audit, sphmp.Context(sc.params) as other:
        ctx.before_first_step()
        st = ctx.rollout(audit, 8, factor=8, audit_every=1, tol=1e-12)
        assert st["fallbacks"] == 1  # ended by it: the state is the audit's
        other.copy_state_from(ctx)
        other.sort()
        shift = _shift(ctx.n, 1e-4)
        got, want = _moved_forces(ctx, shift), _moved_forces(other, shift)
    assert np.abs(want[-1]).max() > 0
    for f, a, b in zip(FIELDS, got, want):
        assert bits_equal(a, b), f
