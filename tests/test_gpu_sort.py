"""The cell sort where its one-pass scan and its counts change course: grids of one and of many scan blocks, out-of-grid
slots spread over more than one group of hash chunks, both cell orders, a cell list asked for twice and after a step
that has cleared the counts. Whole numbers: every array equals a stable sort's."""
import numpy as np
import pytest

import sphmp
from sphmp import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _scene(n, out, order, seed):
    """n fluid particles without walls, a share `out` of them outside the grid, in random order."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    sc = scenes.small_block(seed=seed, n=(side, side, side), nphase=1, dens=(1000.0,), walls=False)
    d, c = sc.disp[:n].copy(), sc.calc[:n].copy()
    d["pos"] = d["pos"][rng.permutation(n)]
    gone = rng.random(n) < out
    d["pos"][gone] = rng.uniform(-50, -20, (int(gone.sum()), 3)).astype(np.float32)
    sc.params.num = sc.params.maxNum = n
    sc.params.cell_order = order
    return sc.params, d, c


def _morton(p, cell):
    x, yz = cell % p.gridres[0], cell // p.gridres[0]
    z, y = yz % p.gridres[2], yz // p.gridres[2]
    code = np.zeros(len(cell), np.int64)
    for b in range(12):
        code |= ((x >> b & 1) << 3 * b) | ((z >> b & 1) << (3 * b + 1)) | ((y >> b & 1) << (3 * b + 2))
    return code


def _lists(ctx):
    return {k: ctx.download_field(f) for k, f in (("midsort", abi.F_MIDSORT), ("mgndx", abi.F_MGNDX), ("mgcell", abi.F_MGCELL),
                                                  ("mgridoff", abi.F_MGRIDOFF), ("mgridcnt", abi.F_MGRIDCNT))}


@pytest.mark.parametrize("order", [abi.CELL_ORDER_LINEAR, abi.CELL_ORDER_MORTON])
@pytest.mark.parametrize("n,out", [(1, 0.0), (1, 1.0), (255, 0.5), (257, 0.0), (4000, 0.2), (150001, 0.0), (150001, 0.01), (150001, 0.7)])
def test_sort_equals_a_stable_sort(n, out, order):
    p, d, c = _scene(n, out, order, n + int(10 * out))
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        for _ in range(2):  # the second hash finds the counts as the first list left them
            ctx.get_particle_index()
            key = ctx.download_field(abi.F_MGCELL)
            ctx.get_grid_list()
        got = _lists(ctx)
        inside = key != abi.GRID_UNDEF
        rank = np.where(inside, _morton(p, key.astype(np.int64)) if order else key.astype(np.int64), 1 << 60)
        perm = np.argsort(rank, kind="stable")
        assert np.array_equal(got["midsort"], perm.astype(np.uint32))
        assert np.array_equal(got["mgcell"], key[perm])
        cnt = np.bincount(key[inside].astype(np.int64), minlength=p.gridtotal)
        assert np.array_equal(got["mgridcnt"], cnt)
        first = np.zeros(p.gridtotal, np.int64)
        sk = key[perm][:int(inside.sum())].astype(np.int64)
        cells, at = np.unique(sk, return_index=True)
        first[cells] = at
        assert np.array_equal(got["mgridoff"], first)
        ndx = np.full(n, abi.GRID_UNDEF, np.uint32)
        ndx[:len(sk)] = np.arange(len(sk)) - first[sk]
        assert np.array_equal(got["mgndx"], ndx)
        ctx.get_grid_list()  # again from the same keys
        again = _lists(ctx)
        for k in got:
            assert np.array_equal(again[k], got[k]), k


@pytest.mark.parametrize("runs", [1, 3, 7, 256])
def test_blocks_that_count_into_many_sums(runs):
    """A block of 256 slots whose particles fall into about `runs` of the grid's ten groups of 4,096 cells: added up
    group by group for four of them, by warps for the rest."""
    n, side = 64000, 40
    sc = scenes.small_block(seed=5, n=(side, side, side), d=0.01, h=0.006, nphase=1, dens=(1000.0,), walls=False)
    p, d, c = sc.params, sc.disp[:n].copy(), sc.calc[:n].copy()
    assert p.gridtotal > 8 * 4096
    rng = np.random.default_rng(runs)
    piece = max(1, 256 // runs)  # stretches of the sorted order, shuffled
    y = np.argsort(d["pos"][:, 1], kind="stable")
    d["pos"] = d["pos"][np.concatenate([y[k * piece:(k + 1) * piece] for k in rng.permutation(-(-n // piece))])]
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        ctx.get_particle_index()
        key = ctx.download_field(abi.F_MGCELL).astype(np.int64)
        ctx.get_grid_list()
        got = _lists(ctx)
    assert (key != abi.GRID_UNDEF).all()
    assert np.array_equal(got["midsort"], np.argsort(key, kind="stable").astype(np.uint32))
    assert np.array_equal(got["mgridcnt"], np.bincount(key, minlength=p.gridtotal).astype(np.int32))
    assert np.array_equal(got["mgcell"], np.sort(key).astype(np.uint32))


@pytest.mark.parametrize("order", [abi.CELL_ORDER_LINEAR, abi.CELL_ORDER_MORTON])
@pytest.mark.parametrize("graph", [False, True])
def test_list_after_a_step(graph, order):
    p, d, c = _scene(70000, 0.3, order, 5)
    with sphmp.Context(p) as ctx:
        ctx.upload_aos(d, c)
        ctx.step(1, abi.SCHEDULE_FUSED, use_graph=graph)
        want = _lists(ctx)
        ctx.get_grid_list()
        got = _lists(ctx)
        for k in want:
            assert np.array_equal(got[k], want[k]), k
        # and the next step's sort is that of a context that never asked
        ctx.get_particle_index()
        ctx.step(1, abi.SCHEDULE_FUSED, use_graph=graph)
        got = _lists(ctx)
        with sphmp.Context(p) as other:
            other.upload_aos(d, c)
            other.step(2, abi.SCHEDULE_FUSED, use_graph=graph)
            for k, v in _lists(other).items():
                assert np.array_equal(got[k], v), k
