"""The corrector network at the edges of its kernels' work: a tile is 128 rows, the
forward pass has four tiles in flight on each SM, and the training pass
accumulates over the tiles of an SM."""
import numpy as np
import pytest
import torch

import sphmp
from oracle import learned as OL

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda")


def _rows(tiles, extra):
    """``tiles`` per SM, ``extra`` rows more or less."""
    return max(1, 128 * tiles * torch.cuda.get_device_properties(0).multi_processor_count + extra)


def _net(seed, batch):
    rng = np.random.default_rng(seed)
    p = OL.init_params(seed)
    shift = (rng.standard_normal(48) * 0.1).astype(np.float32)
    scale = (0.5 + rng.random(48)).astype(np.float32)
    cor = sphmp.Corrector(max_batch=batch)
    cor.set_params(p)
    cor.set_normalisation(shift, scale, np.ones(4, np.float32))
    return cor, p, shift, scale, rng


@pytest.mark.parametrize("tiles,extra", [(0, 1), (0, 127), (0, 128), (0, 129), (1, -1), (1, 0), (1, 1), (2, -129), (2, 0),
                                         (2, 1), (4, 1), (5, 77)])
def test_forward_rows_do_not_depend_on_the_size(built, tiles, extra):
    """A row's outputs take the same operations in the same order wherever its tile
    runs, so they are equal bit for bit to the same rows among many others;
    the rows behind the last stay untouched."""
    n, big = _rows(tiles, extra) if tiles else extra, _rows(6, 0)
    cor, p, shift, scale, rng = _net(8, 0)
    x = torch.from_numpy(rng.standard_normal((big, 48)).astype(np.float32)).to(DEV)
    ref = torch.empty((big, 4), dtype=torch.float32, device=DEV)
    cor.forward(x, ref)
    y = torch.full((n + 64, 4), 7.0, dtype=torch.float32, device=DEV)
    cor.forward(x[:n], y[:n])
    cor.sync()
    assert torch.equal(y[:n], ref[:n]) and bool((y[n:] == 7.0).all())
    cor.close()


@pytest.mark.parametrize("tiles,extra", [(0, 128), (0, 256), (1, -128), (1, 0), (1, 128), (2, 128)])
def test_gradients_at_the_edges_of_a_round(built, tiles, extra):
    """Against the oracle, as at other sizes: the bf16 roundings of the operands are
    the oracle's, a rare one falls to the other side (the hardware tanh)."""
    batch = _rows(tiles, extra) if tiles else extra
    cor, p, shift, scale, rng = _net(9, batch)
    X = rng.standard_normal((batch, 48)).astype(np.float32)
    T = rng.standard_normal((batch, 4)).astype(np.float32)
    g, loss = cor.gradients(torch.from_numpy(X).to(DEV), torch.from_numpy(T).to(DEV))
    gr, lr = OL.mlp_backward(p, shift, scale, X, T)
    assert abs(loss - lr) <= 1e-5 * lr
    G, R = OL.unpack(g), OL.unpack(gr)
    for k in R:
        assert np.linalg.norm(G[k] - R[k]) <= 1e-3 * np.linalg.norm(R[k]), k
    # the same rows twice: every weight gradient is the same, to the order of the FP32 sums
    if 2 * batch <= _rows(2, 0):
        c2 = sphmp.Corrector(max_batch=2 * batch)
        c2.set_params(p)
        c2.set_normalisation(shift, scale, np.ones(4, np.float32))
        g2, loss2 = c2.gradients(torch.from_numpy(np.concatenate([X, X])).to(DEV),
                                 torch.from_numpy(np.concatenate([T, T])).to(DEV))
        assert abs(loss2 - loss) <= 1e-5 * loss
        assert np.linalg.norm(g2 - g) <= 1e-5 * np.linalg.norm(g)
        c2.close()
    cor.close()
