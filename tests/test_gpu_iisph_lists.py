"""The IISPH passes' list walks and shared cell scans at the sizes and states where they change course: fewer
particles than one warp's group, lists beyond their 256 entries (the walk searches the cells), positions that
moved since the sort, lists overwritten by another pass or missing, the Morton cell order, and a solve that ends
inside a batch of queued iterations. Against the oracle's restatement of the reference's kernels on identical
inputs; every sum has at most a few hundred FP32 terms of one sign or with the oracle's own cancellation, so the
fields agree within the 1e-5 of the other IISPH tests."""
import numpy as np
import pytest

import sphmp
from helpers import device_ctx, download_state, field_err, in_grid_fluid, oracle_state, upload_state_fields
from oracle import oracle as O
from sphmp import abi, scenes

pytestmark = pytest.mark.gpu

RTOL = 1e-5

SCENES = {
    "one": dict(n=(1, 1, 1)), "seven": dict(n=(7, 1, 1)), "nine": dict(n=(3, 3, 1)), "ragged": dict(n=(11, 7, 5)),
    "no_walls": dict(n=(9, 8, 7), walls=False), "overflow": dict(n=(16, 16, 16), d=0.02 / 4.2, h=0.02),
    "scaled": dict(n=(9, 8, 7), simscale=0.5),
}


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _pair(name):
    sc = scenes.small_block(seed=61, nphase=2, eos=abi.EOS_TAIT, velocity_scale=0.3, dens=(1000.0, 800.0),
                            multiphase=0, **SCENES[name])
    s = oracle_state(sc)
    O.before_first_step(sc.params, s)
    ctx = device_ctx(sc)
    ctx.before_first_step()
    return sc.params, s, ctx


def _check(ctx, s, names):
    g, f = download_state(ctx), in_grid_fluid(s)
    for k in names:
        assert field_err(g[k][f], getattr(s, k)[f], floor=1e-3) < RTOL, k


@pytest.mark.parametrize("name", list(SCENES))
def test_passes(name):
    p, s, ctx = _pair(name)
    O.call("orc_iisph_density", p, s)
    ctx.iisph_density()
    _check(ctx, s, ["dens"])
    O.call("orc_iisph_predict", p, s)
    ctx.iisph_predict_advection()
    _check(ctx, s, ["veleval"])
    for _ in range(2):
        O.call("orc_iisph_iteration", p, s)
        ctx.iisph_pressure_iteration()
        _check(ctx, s, ["pressure", "accel"])
    ctx.close()


@pytest.mark.parametrize("name", ["ragged", "overflow"])
def test_moved_without_a_sort(name):
    p, s, ctx = _pair(name)
    rng = np.random.default_rng(5)
    s.pos[s.type == 0] += rng.uniform(-2e-3, 2e-3, (int((s.type == 0).sum()), 3)).astype(np.float32)
    upload_state_fields(ctx, s, ["pos"])
    O.call("orc_iisph_density", p, s)
    O.call("orc_iisph_predict", p, s)
    O.call("orc_iisph_iteration", p, s)
    ctx.iisph_density()
    ctx.iisph_predict_advection()
    ctx.iisph_pressure_iteration()
    _check(ctx, s, ["dens", "veleval", "pressure", "accel"])
    ctx.close()


def test_lists_missing_or_overwritten():
    """Predict and iterate without an IISPH density since the lists were last written by another pass."""
    p, s, ctx = _pair("ragged")
    O.call("orc_iisph_density", p, s)
    ctx.compute_pressure()  # the density pass writes lists of its own into the same storage
    ctx.iisph_density()
    ctx.upload_field(abi.F_PRESSURE, s.pressure)
    dens = download_state(ctx)["dens"]
    ctx.compute_pressure()
    ctx.iisph_density()
    assert np.array_equal(download_state(ctx)["dens"], dens)
    ctx.upload_field(abi.F_PRESSURE, s.pressure)
    O.call("orc_iisph_predict", p, s)
    ctx.iisph_predict_advection()
    ctx.upload_field(abi.F_POS, download_state(ctx)["pos"])  # same positions, the lists are dropped
    O.call("orc_iisph_iteration", p, s)
    ctx.iisph_pressure_iteration()
    _check(ctx, s, ["veleval", "pressure", "accel"])
    ctx.close()


def test_morton_matches_linear():
    out = []
    for order in (abi.CELL_ORDER_LINEAR, abi.CELL_ORDER_MORTON):
        sc = scenes.dam_break_2phase(seed=8, n_side=12, box=0.24, eos=abi.EOS_TAIT, multiphase=0)
        sc.params.cell_order = order
        ctx = device_ctx(sc)
        ctx.before_first_step()
        its, _ = ctx.step_iisph(1, tol=0.0, max_iter=3)
        g = download_state(ctx)
        out.append({k: g[k][np.argsort(g["bornid"])] for k in ("pos", "vel", "pressure", "dens")})
        ctx.close()
    for k in out[0]:
        assert field_err(out[1][k], out[0][k]) < RTOL, k


def test_solve_ends_inside_a_batch():
    """A tolerance that the residue of iteration k meets for the first time ends the solve after k iterations, with
    the state and the residues of that iteration, although more iterations were queued."""
    p, s, ctx = _pair("ragged")
    ctx.iisph_density()
    ctx.iisph_predict_advection()
    res = [ctx.iisph_pressure_iteration() for _ in range(12)]
    mean = np.array([r[1] for r in res])
    first = [k for k in range(2, 12) if mean[k] < mean[1:k].min()]
    assert first, mean
    k = first[0]
    zero = np.zeros_like(s.pressure)
    ctx.upload_field(abi.F_PRESSURE, zero)  # the iterate starts from half the stored pressure: the scene's zero again
    ctx.iisph_predict_advection()
    it, r = ctx.iisph_pressure_solve(0.5 * (mean[k] + mean[1:k].min()), 2, 12)
    assert it == k + 1
    assert abs(r[1] - mean[k]) <= 1e-6 * mean[k] and abs(r[0] - res[k][0]) <= 1e-6 * abs(res[k][0])
    got = download_state(ctx)["pressure"]
    ctx.upload_field(abi.F_PRESSURE, zero)
    ctx.iisph_predict_advection()
    for _ in range(k + 1):
        ctx.iisph_pressure_iteration()
    assert field_err(download_state(ctx)["pressure"], got) < 1e-6
    ctx.close()
