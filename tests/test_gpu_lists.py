"""The bucket density pass and the list walks where their shares change: windows of every size that shares the lanes
of a warp differently (1 to 33 members of one h-subcell, boundary particles among them), candidate sequences around
one staged block (256) and beyond, and the particle counts at which a list walk takes eight, four, two or one lane a
particle. Density, forces, drift velocities and fractions after one fused step against the FP32 oracle, with the
tolerance of the other parity tests (1e-5 of the largest value: sums of at most a few hundred FP32 terms)."""
import numpy as np
import pytest

import sphmp
from helpers import UNDEF, device_ctx, download_state, field_err, oracle_state
from oracle import oracle as O
from sphmp import abi, scenes

pytestmark = pytest.mark.gpu

RTOL = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    sphmp.load()


def _step_matches(sc, window=0):
    sc.params.bucket_window = window
    s = oracle_state(sc)
    O.before_first_step(sc.params, s)
    ctx = device_ctx(sc)
    ctx.before_first_step()
    O.step(sc.params, s, abi.SCHEDULE_FUSED, 1)
    ctx.step(1, abi.SCHEDULE_FUSED)
    ctx.sync()
    g = download_state(ctx)
    ctx.close()
    assert np.array_equal(g["midsort"], s.midsort)
    f = (s.type == 0) & (s.mgcell != UNDEF)
    for k in ("dens", "accel", "drift", "alpha", "vel"):
        # (field_err leaves equal entries out of its scale; most fractions equal exactly 0 or 1)
        assert field_err(g[k][f], getattr(s, k)[f], floor=1.0 if k == "alpha" else 0.0) < RTOL, k


def _cluster(members, around, seed):
    """`members` particles in one h-subcell and `around` in each of the 26 others about it; light ones, so that the
    densities stay near the rest density. Some of them are boundary particles."""
    h = 0.02
    per = [members if (x, y, z) == (1, 1, 1) else around for x in range(3) for y in range(3) for z in range(3)]
    n = sum(per)
    side = int(np.ceil(n ** (1 / 3)))
    sc = scenes.small_block(seed=seed, n=(side, side, side), d=h / 2, h=h, nphase=3, walls=False, eos=abi.EOS_LINEAR,
                            dens=(1000.0, 900.0, 800.0), velocity_scale=0.1)
    p = sc.params
    rng = np.random.default_rng(seed)
    gmin, sub = np.array(p.gridmin[:3]), h / p.simscale
    corner = gmin + sub * (2 * np.array([2, 2, 2]) - 1)  # subcells about the first one of cell (2, 2, 2)
    pos = np.concatenate([corner + sub * (np.array([x, y, z]) + rng.uniform(0.02, 0.98, (k, 3))) for k, (x, y, z) in
                          zip(per, [(x, y, z) for x in range(3) for y in range(3) for z in range(3)])])
    d, c = sc.disp[:n].copy(), sc.calc[:n].copy()
    d["pos"] = pos.astype(np.float32)[rng.permutation(n)]
    c["mass"] *= np.float32(8.0 * 27.0 / n)
    wall = rng.random(n) < 0.15
    d["type"][wall] = abi.TYPE_BOUNDARY
    c["restdens"][wall], c["visc"][wall], c["vel"][wall], c["veleval"][wall] = 1000.0, p.bvisc, 0.0, 0.0
    c["dens"][wall] = c["mass"][wall] / 1000.0
    p.num = p.maxNum = n
    return scenes.Scene(p, d, c, int((~wall).sum()), int(wall.sum()))


@pytest.mark.parametrize("members", [1, 2, 3, 5, 8, 9, 11, 16, 17, 31, 32, 33, 70])
def test_window_sizes(members):
    _step_matches(_cluster(members, 4, 80 + members))


@pytest.mark.parametrize("members", [17, 25, 31, 32])
def test_one_lane_a_member(members):
    """Windows of more than 16 members (not the default)."""
    _step_matches(_cluster(members, 4, 700 + members), 32)


@pytest.mark.parametrize("around", [0, 1, 9, 10, 19, 20, 40])
def test_sequence_lengths(around):
    _step_matches(_cluster(6, around, 200 + around))


@pytest.mark.parametrize("members,around", [(4, 4), (5, 4), (8, 8), (9, 8), (16, 16), (17, 16), (32, 32), (33, 32)])
def test_cell_sort_sizes(members, around):
    """A cell of members + 7 around particles: 32, 33, 64, 65, 128, 129, 256 and 257, where a lane of the cell sort
    holds one, two, four or eight of them, or a block sorts the cell."""
    _step_matches(_cluster(members, around, 500 + members))


@pytest.mark.parametrize("window", [8, 16, 32])
def test_window_parameter(window):
    _step_matches(_cluster(40, 12, 300), window)


@pytest.mark.parametrize("lattice", [(24, 16, 24), (30, 24, 32), (60, 40, 60), (96, 64, 80)])
def test_walk_lanes(lattice):
    """About 22 K, 46 K, 209 K and 625 K slots: eight, four, two lanes and one lane a particle."""
    d = 0.005
    _step_matches(scenes.blobs_3phase(seed=9, lattice=lattice, box=(2 * lattice[0] * d, 2 * lattice[1] * d, lattice[2] * d),
                                      n_blobs=16))
