"""catalog.positions where its faster arithmetic could round another way than the reference's
FP64 chain: shifts that put a float32 sum on or next to a tie, cancelling, huge, tiny, zero
and non-finite values, both signs of hz, ragged sizes and unaligned catalogues.  Bit-identical
to the oracle."""
import numpy as np
import pytest

from oracle import pbi4_oracle as O
from pbi4_gb300 import catalog

pytestmark = pytest.mark.gpu

LOS = [([0.0, 0.0, 1.0], 130.8, 0.5), ([0.6, -0.48, 0.64], -71.3, 0.0), ([1e-3, 7.0, 0.0], 3.3e4, 2.75)]


def _nasty(dtype, n, los, hz, z, mode, seed):
    rng = np.random.default_rng(seed)
    box = 1000.0
    pos = rng.uniform(-0.3 * box, 1.3 * box, (n, 3))
    c = np.array(los) * ((1 + z) / hz if mode else 1.0)
    vel = rng.normal(0.0, 500.0, (n, 3))
    pos, vel = pos.astype(dtype), vel.astype(dtype)
    half = (np.spacing(np.abs(pos)) / 2).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore"):
        tie = np.where(c != 0, half / c, 0.0)  # pos + shift on a tie
        kill = np.where(c != 0, -pos / c, 0.0)  # pos + shift near zero
    k = rng.integers(-3, 4, (n, 3)) * rng.choice([1.0, 1e-3, 1e-6], (n, 3))
    pick = rng.integers(0, 6, (n, 3))
    vel = np.where(pick == 0, (tie * rng.choice([1, -1, 3, -5], (n, 3))).astype(dtype), vel)
    vel = np.where(pick == 1, (tie * (1 + k * np.finfo(dtype).eps)).astype(dtype), vel)
    vel = np.where(pick == 2, (kill * (1 + k * 1e-7)).astype(dtype), vel)
    for j, (p, v) in enumerate([(0, 0), (-0.0, -0.0), (0, 1e-30), (1e-38, 1e-38), (1e30, 1), (5, 1e30), (np.inf, 1),
                                (5, np.inf), (np.nan, 1), (5, np.nan), (5, -np.inf), (box, 0), (-box, 0), (2 * box, 0),
                                (3 * box, 0), (-5 * box, 3), (1e-45, 0), (box / 3, -1e-45)]):
        if j < n:
            pos[j, j % 3] = pos[j, (j + 1) % 3] = p
            vel[j, j % 3] = v
    return pos, vel, box


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("los,hz,z", LOS)
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 33, 511, 513, 40961])
def test_catalogue_rounding(dtype, los, hz, z, mode, n):
    import torch
    pos, vel, box = _nasty(dtype, n, los, hz, z, mode, n + mode)
    with np.errstate(all="ignore"):
        ref = O.catalogue_positions(pos, vel, los, hz, z, box=box, rsd_mode=mode)
        ref0 = O.catalogue_positions(pos, box=box)
    # a catalogue that starts one row into its storage: rows are contiguous, 16 bytes are not
    tp, tv = (torch.from_numpy(np.concatenate([a[:1], a])).cuda()[1:] for a in (pos, vel))
    got = catalog.positions(tp, vel=tv, los=los, hz=hz, z=z, box=box, rsd_mode=mode).cpu().numpy()
    np.testing.assert_array_equal(got, ref)
    np.testing.assert_array_equal(catalog.positions(pos, box=box).cpu().numpy(), ref0)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("box", [1.0, 3.0, 677.7, 0.1, 1e-200, 1e35])
def test_catalogue_boxes(dtype, box):
    if dtype == np.float32 and box < 1e-30:
        box = 1e-30
    pos = (np.random.default_rng(3).uniform(-0.9, 1.9, (5000, 3)) * box).astype(dtype)
    with np.errstate(all="ignore"):
        ref = O.catalogue_positions(pos, box=box)
    np.testing.assert_array_equal(catalog.positions(pos, box=box).cpu().numpy(), ref)
