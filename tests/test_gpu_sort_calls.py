"""The sort called in parts, with other calls between the parts: the cell list is made from the keys of the last hash
whatever was done since. Whole numbers: every array equals a stable sort's."""
import numpy as np
import pytest

import sphmp
from helpers import bits_equal, device_ctx
from sphmp import abi, scenes
from test_gpu_sort import _lists, _morton, _scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _expect(p, key, order):
    """The lists of a stable sort by the cell order."""
    n, inside = len(key), key != abi.GRID_UNDEF
    k = key.astype(np.int64)
    perm = np.argsort(np.where(inside, _morton(p, k) if order else k, 1 << 60), kind="stable")
    sk = k[perm][:int(inside.sum())]
    cells, at = np.unique(sk, return_index=True)
    first = np.zeros(p.gridtotal, np.int64)
    first[cells] = at
    ndx = np.full(n, abi.GRID_UNDEF, np.uint32)
    ndx[:len(sk)] = np.arange(len(sk)) - first[sk]
    return {"midsort": perm, "mgcell": key[perm], "mgndx": ndx, "mgridoff": first,
            "mgridcnt": np.bincount(k[inside], minlength=p.gridtotal)}


def _check(ctx, p, key, order):
    got = _lists(ctx)
    for k, v in _expect(p, key, order).items():
        assert np.array_equal(got[k], v), k


LINEAR, MORTON = abi.CELL_ORDER_LINEAR, abi.CELL_ORDER_MORTON


@pytest.mark.parametrize("steps", [("hash", MORTON, "list"), ("hash", LINEAR, "list"), ("hash", "list", MORTON, "list", LINEAR, "list"),
                                   ("step", LINEAR, "list"), ("step", MORTON, "list")])
@pytest.mark.parametrize("first", [LINEAR, MORTON])
def test_cell_order_changes_between_the_calls(first, steps):
    p, d, c = _scene(150001, 0.01, first, 3)
    assert p.gridtotal > 4 * 4096  # several blocks of the scan
    c["bornid"] = np.arange(p.num)
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        if steps[0] == "step":  # the step's own sort has used the counts up
            ctx.step(1, abi.SCHEDULE_FUSED)
            key = np.empty(p.num, np.uint32)
            key[ctx.download_field(abi.F_MIDSORT)] = ctx.download_field(abi.F_MGCELL)
        else:
            ctx.get_particle_index()
            key = ctx.download_field(abi.F_MGCELL)
        order = first
        for s in steps[1:]:
            if s == "list":
                ctx.get_grid_list()
                _check(ctx, p, key, order)
            else:
                order = s
                q = ctx.get_params()
                q.cell_order = order
                ctx.set_params(q)
        ctx.rearrange_data()
        assert np.array_equal(np.sort(ctx.download_field(abi.F_BORNID)), np.arange(p.num))


def _dense(per):
    """`per` particles in each h-subcell of four cells along every axis, in a grid with no room to spare."""
    h, sub = 0.02, 8
    sc = scenes.small_block(seed=per, n=(16, 16, 16), d=h / 2, h=h, nphase=2, walls=False, eos=abi.EOS_LINEAR,
                            box=(sub * h, sub * h, sub * h), dens=(1000.0, 900.0), velocity_scale=0.1)
    p, n = sc.params, per * sub ** 3
    rng = np.random.default_rng(per)
    d, c = sphmp.record_arrays(n)
    src = rng.integers(0, len(sc.disp), n)
    d[:], c[:] = sc.disp[src], sc.calc[src]
    cell = np.repeat(np.stack(np.meshgrid(*[np.arange(sub)] * 3, indexing="ij"), -1).reshape(-1, 3), per, axis=0)
    at = np.array(p.gridmin[:3]) + 2 * h / p.simscale  # the first inner cell
    d["pos"] = (at + (cell + rng.uniform(0.02, 0.98, (n, 3))) * h / p.simscale)[rng.permutation(n)]
    c["mass"] *= np.float32(8.0 / per)
    p.num = p.maxNum = n
    return scenes.Scene(p, d, c, n, 0)


def _state(ctx):
    return {f: ctx.download_field(f) for f in (abi.F_MIDSORT, abi.F_POS, abi.F_DENS, abi.F_PRESSURE, abi.F_ACCEL)}


@pytest.mark.parametrize("twice", ["counts", "list"])
def test_cells_listed_twice_from_one_hash(twice):
    """The cells scanned for uploaded counts (the same ones) or listed, and listed again: occupied cells, large cells
    and member windows are counted once. A cell holds 320 particles, a particle has about 170 neighbours."""
    sc = _dense(40)
    got = []
    for again in (False, True):
        with device_ctx(sc) as ctx:
            ctx.before_first_step()
            ctx.get_particle_index()
            if again and twice == "counts":
                ctx.upload_field(abi.F_MGRIDCNT, ctx.download_field(abi.F_MGRIDCNT))
            elif again:
                ctx.get_grid_list()
            ctx.get_grid_list()
            ctx.rearrange_data()
            ctx.compute_pressure()
            ctx.compute_force()
            got.append(_state(ctx))
    for f, v in got[0].items():
        assert bits_equal(got[1][f], v), f


def test_list_between_density_and_force():
    """The queue of particles with many neighbours outlives a cell list made between the passes."""
    sc = _dense(40)
    got = []
    for again in (False, True):
        with device_ctx(sc) as ctx:
            ctx.before_first_step()
            ctx.sort()
            ctx.compute_pressure()
            if again:
                ctx.get_grid_list()
            ctx.compute_force()
            got.append(_state(ctx))
    assert bits_equal(got[1][abi.F_ACCEL], got[0][abi.F_ACCEL])
    assert np.abs(got[0][abi.F_ACCEL]).max() > 0


def _captured(ctx, calls):
    """`calls` on the context's stream as a caller's own graph; nothing of it has run yet."""
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        calls()
        graph.capture_end()

    def replay():
        with torch.cuda.stream(stream):
            graph.replay()
    return replay


@pytest.mark.parametrize("before", ["calls", "step", "replayed steps"])
@pytest.mark.parametrize("order", [LINEAR, MORTON])
def test_a_callers_capture_of_the_sort(order, before):
    """Two sorts captured by the caller and replayed, with the library's own sorts, steps and lists in between: what a
    replay counts does not depend on what ran before it."""
    p, d, c = _scene(70000, 0.3, order, 6)
    c["bornid"] = np.arange(p.num)
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        if before == "calls":
            ctx.sort()
        else:
            ctx.step(2, abi.SCHEDULE_FUSED, use_graph=before != "step")
        replay = _captured(ctx, lambda: (ctx.sort(), ctx.sort()))
        for k in range(4):
            replay()
            if k:  # the first replays follow one another
                ctx.sync()
                key = ctx.download_field(abi.F_MGCELL)  # sorted: the next sort leaves the order
                _check(ctx, p, key, order)
                assert np.array_equal(np.sort(ctx.download_field(abi.F_BORNID)), np.arange(p.num))
            if k == 1:
                ctx.get_particle_index()
            elif k == 2:
                ctx.step(2, abi.SCHEDULE_FUSED)
        ctx.get_grid_list()
        _check(ctx, p, key, order)
        ctx.sync()


def test_a_callers_capture_of_a_step():
    p, d, c = _scene(70000, 0.3, LINEAR, 7)
    c["bornid"] = np.arange(p.num)
    fields = (abi.F_BORNID, abi.F_POS, abi.F_VEL, abi.F_ACCEL, abi.F_MGRIDCNT)
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        ctx.step(1, abi.SCHEDULE_FUSED, use_graph=False)
        replay = _captured(ctx, lambda: ctx.step(1, abi.SCHEDULE_FUSED, use_graph=False))
        replay()
        ctx.get_particle_index()
        replay()
        ctx.step(2, abi.SCHEDULE_FUSED, use_graph=True)
        replay()
        ctx.sync()
        got = [ctx.download_field(f) for f in fields]
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        ctx.step(6, abi.SCHEDULE_FUSED)
        ctx.sync()
        want = [ctx.download_field(f) for f in fields]
    for f, a, b in zip(fields, got, want):
        assert bits_equal(a, b), f


@pytest.mark.parametrize("order", [LINEAR, MORTON])
def test_a_callers_capture_of_the_list(order):
    """The list alone, replayed after steps that have cleared the counts and after ones that have not."""
    p, d, c = _scene(70000, 0.3, order, 8)
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        ctx.sort()
        ctx.get_particle_index()
        replay = _captured(ctx, ctx.get_grid_list)
        for use_graph in (None, True, False, True, True):
            if use_graph is not None:
                ctx.step(1, abi.SCHEDULE_FUSED, use_graph=use_graph)
                want = _lists(ctx)
            replay()
            ctx.sync()
            if use_graph is not None:
                got = _lists(ctx)
                for k in want:
                    assert np.array_equal(got[k], want[k]), (k, use_graph)


def test_list_after_uploaded_counts():
    """A list is made from the keys, whatever counts the caller has put in."""
    p, d, c = _scene(70000, 0.3, LINEAR, 9)
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        ctx.get_particle_index()
        key = ctx.download_field(abi.F_MGCELL)
        cnt = np.zeros(p.gridtotal, np.int32)
        cnt[100:200] = 7
        ctx.upload_field(abi.F_MGRIDCNT, cnt)
        ctx.get_grid_list()
        _check(ctx, p, key, LINEAR)
        ctx.step(1, abi.SCHEDULE_FUSED)
        ctx.upload_field(abi.F_MGRIDCNT, cnt)
        ctx.get_grid_list()
        _check(ctx, p, key, LINEAR)
