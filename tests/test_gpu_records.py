"""Record transfers and boundary volumes at the edges of a warp's share (32 records, 8 particles): the records come
back byte for byte (a copy), the volumes against the FP64 oracle with at most four times the FP32 oracle's own error
(or 2e-7, three roundings of the result)."""
import numpy as np
import pytest
import torch

import sphmp
from helpers import device_ctx, oracle_state
from oracle import oracle as O
from sphmp import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 1000])
def test_round_trip(n):
    sc = scenes.small_block(seed=71, n=(16, 16, 16), nphase=3, walls=False, velocity_scale=0.5)
    rng = np.random.default_rng(n)
    d, c = sc.disp[:n].copy(), sc.calc[:n].copy()
    d["color"] = rng.random((n, 4))
    c["accel"], c["veleval"] = rng.random((n, 3)), rng.random((n, 3))
    c["pressure"], c["dens"], c["visc"] = rng.random(n), rng.random(n), rng.random(n)
    c["bornid"] = rng.permutation(n)
    guard = 7  # records past the end keep their bytes
    with sphmp.Context(sc.params) as ctx:
        ctx.upload_aos(d, c)
        out = sphmp.record_arrays(n + guard)
        for a in out:
            a.view(np.uint8)[:] = 0xA5
        ctx.download_aos(n, out=out)
        assert out[0][:n].tobytes() == d.tobytes()
        for k in ("vel", "veleval", "pressure", "dens", "restdens", "mass", "visc", "bornid", "accel"):
            assert np.array_equal(out[1][k][:n], c[k]), k
        for k in ("deformGrad", "stress", "B", "solidG", "solidK", "X", "invA"):
            assert not out[1][k][:n].any(), k
        for a in out:
            assert (a[n:].view(np.uint8) == 0xA5).all()
        only = ctx.download_aos(n, calc=False)
        assert only.tobytes() == d.tobytes()


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n", [1, 33, 1000])
def test_upload_reads_no_solid_fields(n, pinned):
    """Only the first 64 bytes of a calculation record go up; what the others hold does not matter, for an upload,
    an append and a state copy (whole records on the device) alike."""
    sc = scenes.small_block(seed=73, n=(16, 16, 16), nphase=3, walls=False, velocity_scale=0.5)
    rng = np.random.default_rng(n)
    d, c = sc.disp[:2 * n].copy(), sc.calc[:2 * n].copy()
    want = c.copy()
    c.view(np.uint8).reshape(2 * n, 224)[:, 60:] = rng.integers(0, 256, (2 * n, 164), dtype=np.uint8)
    if pinned:
        d, c = (torch.from_numpy(a.view(np.uint8)).pin_memory().numpy().view(a.dtype) for a in (d, c))
    with sphmp.Context(sc.params) as ctx, sphmp.Context(sc.params) as other:
        ctx.upload_aos(d[:n], c[:n])
        ctx.emit_aos(d[n:], c[n:], n, 2 * n)
        ctx.sync()
        other.copy_state_from(ctx)
        for x in (ctx, other):
            out = x.download_aos()
            assert out[0].tobytes() == d.tobytes()
            for k in ("vel", "veleval", "pressure", "dens", "restdens", "mass", "visc", "bornid", "accel"):
                assert np.array_equal(out[1][k], want[k]), k


@pytest.mark.parametrize("kind", [(1, 1, 1), (3, 2, 5), (9, 7, 6)])
@pytest.mark.parametrize("order", [abi.CELL_ORDER_LINEAR, abi.CELL_ORDER_MORTON])
def test_boundary_volume(kind, order):
    sc = scenes.small_block(seed=72, n=kind, nphase=1, dens=(1000.0,))
    ref = {}
    for t in (np.float32, np.float64):
        s = oracle_state(sc, t)
        O.before_first_step(sc.params, s)
        b = (s.type == 1) & (s.mgcell != abi.GRID_UNDEF)
        ref[t] = dict(zip(s.bornid[b].tolist(), s.dens[b].astype(np.float64)))
    sc.params.cell_order = order
    ctx = device_ctx(sc)
    ctx.before_first_step()
    got = dict(zip(ctx.download_field(abi.F_BORNID).tolist(), ctx.download_field(abi.F_DENS).astype(np.float64)))
    ctx.close()
    ids = sorted(ref[np.float64])
    assert len(ids) > 100
    v = {k: np.array([d[i] for i in ids]) for k, d in (("g", got), ("f", ref[np.float32]), ("d", ref[np.float64]))}
    err = np.abs(v["g"] / v["d"] - 1).max()
    assert err <= max(4 * np.abs(v["f"] / v["d"] - 1).max(), 2e-7), err
