"""The sort called in parts, with other calls between the parts: the cell list is made from the keys of the last hash
whatever was done since. Whole numbers: every array equals a stable sort's."""
import numpy as np
import pytest

import sphmp
from sphmp import abi
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
